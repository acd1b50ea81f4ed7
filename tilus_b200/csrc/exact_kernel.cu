// Batches of up to 16 rows on tcgen05: C[M, N] = A[M, K] x dequant(Bq[K, N]) with exact weights.
// Serves 5 to 16 rows, and fewer where K is not in whole 512-row blocks or stream_outrun says so, as far as resident_kernel.cu does not
// take them (api.cu, resident_cluster): bfloat16 wherever the stream kernel has not, fp16 mostly wide or deep layers of 9 to 16 rows.
//
// Same product and work split as batch_kernel.cu (weights of 128 columns in tensor memory, equal runs of 128-row
// groups per CTA), but the scale is not applied to the weights.  Every group's product is a sum of its own,
// multiplied by the group's scale in fp32 when it is added to the column's sum - no weight is rounded, as in
// stream_kernel.cu - and the decode shrinks to bit extraction:
//   * fp16 activations: an integer code sits at bit 0 of an fp16 subnormal (value code * 2^-24), a float code
//     in its own fields (decode.cuh, pair_lin_uniform).  The tensor core multiplies these exactly.  The zero
//     point is subtracted by a second set of MMAs whose weight operand is the constant -zero_point * 2^-24,
//     each right behind the 16 rows it belongs to.  With all of them behind the group's products the sums ran up to
//     (code) before they came back to (code - zero point), and the fp32 accumulator lost bits to it: 8 x 4096 x 4096,
//     uint8, activations around 3, 6.3 % of the outputs were not the nearest fp16 value (stream_kernel.cu 3.3 %;
//     now 0.3 %).  Single bits need none of this: (code - 1) is the inverted bit, negated;
//   * bf16 activations: exact bf16 values (pair_exact; bf16 has no room for the subnormal trick).
// That is what decides this kernel's speed: integer, shift and half instructions issue every second cycle
// per SM quadrant on this GPU (measured: LOP3, SHF, PRMT, HFMA2 2.0 cycles, LOP3 + HFMA2 3.7 together, FFMA 1.0),
// and a 128 x 128 group of 4-bit weights costs 112 of them per thread here against 208 with scaled weights.
// The HBM time of such a group is 355 cycles per SM.
//
// Roles of the warps of a CTA (20 of them; one CTA per SM):
//   * warps 0-11 decode, in three sets of four (lane L of a set's four warps is column L of the tile); set s takes
//     the groups s, s + 3, ... of the CTA's run, two operand slots each.  Before a set stores into a slot
//     it reads the sums of the group that was there (16 columns of tensor memory) and adds them, times their
//     scale, to its fp32 sums of the column: one wait serves the slot and the sums.  A set needs about 1200
//     cycles per group, most of them latencies of its barriers and of tensor memory, so their number sets the
//     rate of narrow weights;
//   * four warps finish column tiles: the sets hand over their sums through shared memory, so that the
//     decoding goes on while a tile's last contributions are counted and written;
//   * one warp each (one elected thread) brings the activations, the packed weights, the scales;
//   * one warp owns tensor memory and issues the MMAs: 8 (or 16 with a zero point) per group, one commit.
//
// Measured (4-bit, group 128, 16 rows, a chain of cold launches; stream_kernel.cu before): 28672 x 4096 37.3 -> 20.8 us,
// 8192 x 8192 19.5 -> 14.3, 4096 x 4096 10.2 -> 8.3, against 9.4, 5.4 and 1.4 us of HBM time.  What is left is the start and
// the end of a launch (about 5 us: 640 threads of 91 .. 96 registers leave no room for another GEMM's CTA on the SM, so
// nothing of it lies under the launch before) and the decode's instructions.
//
// Every mbarrier wait is bounded in time; a wait that runs out raises a CTA-wide abort flag, all loops
// leave, the producers give their copies in flight a bounded chance to land, tensor memory is freed and
// the status word of the workspace reports it.
#include <cuda.h>

#include "batch_common.cuh"

#ifndef B200Q_PART
#define B200Q_PART 0
#endif
#ifndef B200Q_NPARTS
#define B200Q_NPARTS 1
#endif

namespace b200q {

constexpr int EXACT_SETS = 3;                // decode sets of four warps
constexpr int EXACT_SPS = 2;                 // operand slots per set
constexpr int EXACT_SLOTS = EXACT_SETS * EXACT_SPS;  // also: activation groups in shared memory
constexpr int EXACT_THREADS = EXACT_SETS * 128 + 256;
constexpr int EXACT_STAGES_MAX = 18;         // 128-row groups in the packed ring (a multiple of the sets)
constexpr uint32_t EXACT_ASTAGE = 16 * 256;  // 16 rows x 128 columns, two swizzled 64-column blocks
// a set's sums of one tile: quads of four rows x 128 columns
__host__ __device__ constexpr uint32_t exact_hand_bytes(int M) { return (uint32_t)((M + 3) / 4) * 2048u; }

struct ExactBarriers {
  uint64_t slot_full[EXACT_SLOTS];
  uint64_t done[EXACT_SLOTS];  // [i]: the MMAs of a group in slot i have completed
  uint64_t a_full[EXACT_SLOTS];
  uint64_t g_full[EXACT_STAGES_MAX], g_empty[EXACT_STAGES_MAX];
  uint64_t hand_full[EXACT_SETS], hand_empty[EXACT_SETS];  // a set's sums of a segment are in shared memory / have been taken
  uint32_t tmem_base;
  volatile int abort_flag;
};
constexpr int EXACT_BARRIERS = (int)(offsetof(ExactBarriers, tmem_base) / 8);
// arrivals that complete a phase of the i-th barrier
__host__ __device__ constexpr int exact_barrier_count(int i) {
  return i < (int)(offsetof(ExactBarriers, done) / 8) ? 4
       : i < (int)(offsetof(ExactBarriers, g_full) / 8) ? 1
       : i < (int)(offsetof(ExactBarriers, g_empty) / 8) ? 2 : 4;
}

template <int VAR, int ACT>
__global__ void __launch_bounds__(EXACT_THREADS, 1)
exact_kernel(const BatchParams p, const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_w) {
  constexpr int B = var_bits(VAR);
  constexpr int BIAS = ACT == 0 ? lin_uniform_bias(VAR) : 0;  // what the constant operand subtracts
  constexpr float F = ACT == 0 ? (lin_uniform_inverted(VAR) ? -1.0f : 1.0f) * (float)(1u << lin_factor_log2(VAR)) : 1.0f;
  constexpr uint32_t WSTAGE = 2048u * B, SSTAGE = 256u;
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  const uint32_t smem_unaligned = (uint32_t)__cvta_generic_to_shared(smem_raw);
  const uint32_t smem_base = (smem_unaligned + 1023u) & ~1023u;
  unsigned char* smem_al = smem_raw + (smem_base - smem_unaligned);
  const int WS = p.stages;
  const uint32_t HAND = exact_hand_bytes(p.M);
  const uint32_t ring_s = smem_base + EXACT_SLOTS * EXACT_ASTAGE;
  const uint32_t scales_s = ring_s + (uint32_t)WS * WSTAGE;
  const uint32_t hand_off = EXACT_SLOTS * EXACT_ASTAGE + (uint32_t)WS * (WSTAGE + SSTAGE);
  const uint32_t bars_off = hand_off + EXACT_SETS * HAND;
  ExactBarriers* bars = reinterpret_cast<ExactBarriers*>(smem_al + bars_off);
  const uint32_t bars_s = smem_base + bars_off;
#define BAR_ADDR(field, i) (bars_s + (uint32_t)offsetof(ExactBarriers, field) + (uint32_t)(i) * 8u)

  const int tid = threadIdx.x, lane = tid & 31;
  const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
  volatile int* abort_flag = &bars->abort_flag;
  // this CTA's run of groups, counted tile by tile over the whole matrix
  const int run0 = batch_run_start(p, blockIdx.x), run1 = batch_run_start(p, blockIdx.x + 1);

  constexpr int W_EPI = EXACT_SETS * 4, W_ACT = W_EPI + 4, W_WEIGHTS = W_EPI + 5, W_MMA = W_EPI + 6;
  // (by the lanes of one warp while the descriptors are on their way, as in batch_kernel.cu)
  if (warp == W_WEIGHTS && lane == 0) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(&tmap_w) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&tmap_a) : "memory");
  }
  if (warp == 0) {
    for (int i = lane; i < EXACT_BARRIERS; i += 32) mbar_init(bars_s + (uint32_t)i * 8u, (uint32_t)exact_barrier_count(i));
    if (lane == 0) bars->abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  __syncthreads();
  // the producers may start; the roles that use tensor memory wait for it below (the previous launch's CTA on
  // this SM may still hold it)
  if (warp == W_MMA) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(
                     bars_s + (uint32_t)offsetof(ExactBarriers, tmem_base))
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    // Only now may the next launch start: a CTA of it that got this SM's tensor memory first would wait for this
    // launch to complete, and this launch for the tensor memory.  (With this order a launch whose CTAs wait for
    // their predecessor never holds tensor memory that the predecessor still has to get, on whatever streams.)
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  }
  if (warp < W_EPI || warp == W_MMA) {
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    asm volatile("bar.sync 1, %0;" ::"n"(EXACT_SETS * 128 + 32) : "memory");
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  }
  const uint32_t tmem = (warp < W_EPI || warp == W_MMA) ? __shfl_sync(0xffffffffu, bars->tmem_base, 0) : 0u;
  // tensor memory: 16 columns of sums per slot, 64 columns of weights per slot, 8 columns of the constant operand
  const uint32_t slots_t = tmem + 16 * EXACT_SLOTS, const_t = slots_t + 64 * EXACT_SLOTS;

  float acc[16];  // decode warps: this column's sums
  if (warp < W_EPI) {
    // ================= decode =================
    const int set = warp >> 2, wq = warp & 3;
    const int nl = wq * 32 + lane;  // lane of tensor memory = column inside the tile
    const uint32_t lane_t = (uint32_t)(wq * 32) << 16;
#pragma unroll
    for (int i = 0; i < 16; ++i) acc[i] = 0.f;
    if (BIAS != 0 && set == 0) {  // the constant operand: seen by the MMAs behind the first slot_full of set 0
      const uint32_t v = dup16(0x8000u | (uint32_t)BIAS);  // -zero_point * 2^-24
      asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %1, %1, %1, %1, %1, %1, %1};" ::"r"(const_t + lane_t),
                   "r"(v)
                   : "memory");
    }
    float sq[EXACT_SPS];  // scales of the groups in the set's slots
    int stage = set;      // the set's stages: set, set + EXACT_SETS, ...
    uint32_t ring_phase = 0, hand_phase = 1;
    const int n_own = (run1 - run0 - set + EXACT_SETS - 1) / EXACT_SETS;
    const bool more = p.M > 4, most = p.M > 8;
    const bool alone = p.cluster <= 1;
    int seg_end = min((run0 / p.G + 1) * p.G, run1);  // of the segment the sums belong to
    int pos = run0 + set;                             // group whose sums are added next
    while (pos >= seg_end && seg_end < run1) seg_end = min(seg_end + p.G, run1);  // (first segments without a group of this set)
    bool good = true;
    for (int i0 = 0; i0 < n_own + EXACT_SPS && good; i0 += EXACT_SPS) {
#pragma unroll
      for (int j = 0; j < EXACT_SPS; ++j) {
        const int i = i0 + j, slot = set + EXACT_SETS * j;
        const bool have = i < n_own;
        if (i >= EXACT_SPS && i - EXACT_SPS < n_own) {
          // the group this slot held: its sums, times its scale
          if (!mbar_wait_abortable(BAR_ADDR(done, slot), (uint32_t)(i / EXACT_SPS - 1) & 1u, abort_flag)) { good = false; break; }
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const uint32_t d_t = tmem + lane_t + (uint32_t)(slot * 16);
          uint32_t v[16];
          tmem_ld_4_async(d_t, v);
          if (more) tmem_ld_4_async(d_t + 4, v + 4);
          if (most) tmem_ld_8_async(d_t + 8, v + 8);
          tmem_ld_wait(v);
#pragma unroll
          for (int q = 0; q < 4; ++q) acc[q] = fmaf(sq[j], __uint_as_float(v[q]), acc[q]);
          if (more) {
#pragma unroll
            for (int q = 4; q < 8; ++q) acc[q] = fmaf(sq[j], __uint_as_float(v[q]), acc[q]);
          }
          if (most) {
#pragma unroll
            for (int q = 8; q < 16; ++q) acc[q] = fmaf(sq[j], __uint_as_float(v[q]), acc[q]);
          }
          if (alone && pos + EXACT_SETS >= seg_end) {  // the set's last group of the column tile: hand the sums over
            if (!mbar_wait_abortable(BAR_ADDR(hand_empty, set), hand_phase, abort_flag)) { good = false; break; }
            hand_phase ^= 1u;
            float4* hand = reinterpret_cast<float4*>(smem_al + hand_off + (uint32_t)set * HAND) + nl;
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              if (q * 4 < p.M) hand[q * 128] = make_float4(acc[4 * q], acc[4 * q + 1], acc[4 * q + 2], acc[4 * q + 3]);
              acc[4 * q] = acc[4 * q + 1] = acc[4 * q + 2] = acc[4 * q + 3] = 0.f;
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(BAR_ADDR(hand_full, set));
            // (segments without a group of this set are passed over)
            do seg_end = min(seg_end + p.G, run1); while (pos + EXACT_SETS >= seg_end && seg_end < run1);
          }
          pos += EXACT_SETS;
        }
        if (have) {
          if (!mbar_wait_abortable(BAR_ADDR(g_full, stage), ring_phase, abort_flag)) { good = false; break; }
          const uint32_t st = ring_s + (uint32_t)stage * WSTAGE;
          unsigned short sb;
          asm volatile("ld.shared.u16 %0, [%1];" : "=h"(sb) : "r"(scales_s + (uint32_t)stage * SSTAGE + (uint32_t)nl * 2u));
          uint32_t w[2][2 * B];
          batch_load_units<B>(st, nl, 0, w[0]);
          if (B <= 4) batch_load_units<B>(st, nl, 1, w[1]);
          sq[j] = (ACT == 0 ? __half2float(__ushort_as_half(sb)) : __uint_as_float((uint32_t)sb << 16)) * F;
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            if (B > 4 && u == 2) batch_load_units<B>(st, nl, 1, w[1]);
            uint32_t out[16];
            if constexpr (ACT == 0) unit_decode_linear_uniform<VAR>(w[u >> 1] + (u & 1) * B, out);
            else unit_decode_exact<VAR, ACT>(w[u >> 1] + (u & 1) * B, out);
            if (u == 3) {  // the stage has been read (its values fed the arithmetic above)
              __syncwarp();
              if (lane == 0) mbar_arrive(BAR_ADDR(g_empty, stage));
            }
            tmem_st_16(slots_t + lane_t + (uint32_t)(slot * 64 + u * 16), out);
          }
          stage += EXACT_SETS;
          if (stage >= WS) { stage = set; ring_phase ^= 1u; }
          asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
          asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
          __syncwarp();
          if (lane == 0) mbar_arrive(BAR_ADDR(slot_full, slot));
        }
      }
    }
  } else if (warp < W_ACT) {
    // ================= column tiles: sums of all sets, to C or to the tile's scratch =================
    const int wq = warp & 3, nl = wq * 32 + lane;
    asm volatile("griddepcontrol.wait;" ::: "memory");  // C and the scratch may still be in use by the previous kernel
    uint32_t phase = 0u;  // bit s: of set s
    bool good = true;
    for (int pos = run0; pos < run1 && good && p.cluster <= 1;) {
      const int tile = pos / p.G, len = min((tile + 1) * p.G, run1) - pos;
      float4 f[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) f[q] = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
      for (int set = 0; set < EXACT_SETS; ++set) {
        if ((set + EXACT_SETS - (pos - run0) % EXACT_SETS) % EXACT_SETS >= len) continue;  // no group of this set
        if (!mbar_wait_abortable(BAR_ADDR(hand_full, set), (phase >> set) & 1u, abort_flag)) { good = false; break; }
        phase ^= 1u << set;
        const float4* hand = reinterpret_cast<const float4*>(smem_al + hand_off + (uint32_t)set * HAND) + nl;
#pragma unroll
        for (int q = 0; q < 4; ++q)
          if (q * 4 < p.M) {
            const float4 x = hand[q * 128];
            f[q].x += x.x; f[q].y += x.y; f[q].z += x.z; f[q].w += x.w;
          }
        __syncwarp();
        if (lane == 0) mbar_arrive(BAR_ADDR(hand_empty, set));
      }
      if (!good) break;
      const bool whole = len == p.G;
      float4* sums = reinterpret_cast<float4*>(p.partial) + (size_t)tile * (p.rows * 32) + nl;
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        if (q * 4 >= p.M) continue;
        if (whole)
          batch_store4<ACT>(p, tile * 128 + nl, lane, q * 4, f[q]);
        else
          asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(sums + q * 128), "f"(f[q].x), "f"(f[q].y),
                       "f"(f[q].z), "f"(f[q].w)
                       : "memory");
      }
      if (!whole) batch_finish<ACT>(p, tile, len, wq, lane, 0, 1);
      pos += len;
    }
  } else if (warp == W_ACT) {
    // ================= TMA producer: activations =================
    if (elect_one()) {
      asm volatile("griddepcontrol.wait;" ::: "memory");
      int stage = 0, n_issued = 0;
      uint32_t phase = 1;  // of the group that held the stage, whose MMAs report on its slot's barrier
      bool good = true;
      int g = run0 % p.G;
      for (int pos = run0; pos < run1; ++pos) {
        if (n_issued >= EXACT_SLOTS && !mbar_wait_abortable(BAR_ADDR(done, stage), phase, abort_flag)) { good = false; break; }
        const uint32_t bar = BAR_ADDR(a_full, stage);
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(EXACT_ASTAGE) : "memory");
#pragma unroll
        for (int h = 0; h < 2; ++h)
          asm volatile(
              "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
              ::"r"(smem_base + (uint32_t)stage * EXACT_ASTAGE + (uint32_t)h * (EXACT_ASTAGE / 2)), "l"(&tmap_a), "r"(bar),
              "r"(g * 128 + h * 64), "r"(0)
              : "memory");
        ++n_issued;
        if (++stage == EXACT_SLOTS) { stage = 0; phase ^= 1u; }
        if (++g == p.G) g = 0;
      }
      if (!good) {  // a copy in flight must not outlive the CTA: a bounded wait for the groups issued last
        for (int i = max(0, n_issued - EXACT_SLOTS); i < n_issued; ++i)
          mbar_wait_bounded(BAR_ADDR(a_full, i % EXACT_SLOTS), (uint32_t)(i / EXACT_SLOTS) & 1u);
      }
    }
  } else if (warp != W_MMA) {
    // ================= TMA producers: packed weights, scales =================
    if (elect_one()) {
      const bool weights = warp == W_WEIGHTS;
      int stage = 0, n_issued = 0;
      uint32_t phase = 1;
      bool good = true;
      int tile = run0 / p.G, g = run0 - tile * p.G;
      const int groups_per_row = p.group / 128;  // 128-row groups per scale row
      int in_row = g % groups_per_row;
      const __half* sc = p.scales + (size_t)(g / groups_per_row) * p.N + tile * 128;
      uint32_t sc_bytes = (uint32_t)min(128, p.N - tile * 128) * 2u;
      for (int pos = run0; pos < run1; ++pos) {
        if (!mbar_wait_abortable(BAR_ADDR(g_empty, stage), phase, abort_flag)) { good = false; break; }
        const uint32_t bar = BAR_ADDR(g_full, stage);
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(weights ? WSTAGE : sc_bytes)
                     : "memory");
        if (weights)  // (pieces past the last column are filled with zeros and count as bytes all the same)
          asm volatile(
              "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
              ::"r"(ring_s + (uint32_t)stage * WSTAGE), "l"(&tmap_w), "r"(bar), "r"(0),
              "r"(batch_swizzled(B) ? g * (2 * B) : g), "r"(tile * 8)
              : "memory");
        else
          asm volatile(
              "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                  scales_s + (uint32_t)stage * SSTAGE),
              "l"(sc), "r"(sc_bytes), "r"(bar)
              : "memory");
        ++n_issued;
        if (++in_row == groups_per_row) { in_row = 0; sc += p.N; }
        if (++g == p.G) {
          g = 0; in_row = 0; ++tile;
          sc = p.scales + tile * 128;
          sc_bytes = (uint32_t)min(128, p.N - tile * 128) * 2u;
        }
        if (++stage == WS) { stage = 0; phase ^= 1u; }
      }
      if (!good) {
        for (int i = max(0, n_issued - WS); i < n_issued; ++i)
          mbar_wait_bounded(BAR_ADDR(g_full, i % WS), (uint32_t)(i / WS) & 1u);
      }
    }
  } else {
    // ================= MMA issuer =================
    if (elect_one()) {
      const uint32_t idesc = umma_idesc<ACT>(16);
      int slot = 0;
      uint32_t phase = 0;
      // the next group's barriers are looked at before this group's MMAs are issued, so that the latency of
      // the looks lies under them; only a group that was not ready then is waited for
      bool ready = false;
      for (int pos = run0; pos < run1; ++pos) {
        if (!ready && (!mbar_wait_abortable(BAR_ADDR(slot_full, slot), phase, abort_flag) ||
                       !mbar_wait_abortable(BAR_ADDR(a_full, slot), phase, abort_flag))) break;
        const int slot1 = slot + 1 == EXACT_SLOTS ? 0 : slot + 1;
        const uint32_t phase1 = phase ^ (slot1 == 0 ? 1u : 0u);
        const bool next0 = mbar_test(BAR_ADDR(slot_full, slot1), phase1);
        const bool next1 = mbar_test(BAR_ADDR(a_full, slot1), phase1);
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint64_t bdesc = umma_smem_desc(smem_base + (uint32_t)slot * EXACT_ASTAGE);
        const uint32_t a_t = slots_t + (uint32_t)(slot * 64), d_t = tmem + (uint32_t)(slot * 16);
        // the zero point of every 16 rows right behind their products: the running sum stays a sum of (code - zero point)
#pragma unroll
        for (int i = 0; i < (BIAS != 0 ? 16 : 8); ++i) {
          const int ks = BIAS != 0 ? i >> 1 : i;
          const uint32_t op_t = BIAS != 0 && (i & 1) ? const_t : a_t + (uint32_t)(ks * 8);
          const uint64_t bd = bdesc + (uint64_t)((ks & 3) * 2) + ((ks & 4) ? EXACT_ASTAGE >> 5 : 0u);
          if (i == 0)
            asm volatile(
                "{\n\t.reg .pred p;\n\t"
                "setp.ne.b32 p, 0, 0;\n\t"
                "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
                ::"r"(d_t), "r"(op_t), "l"(bd), "r"(idesc)
                : "memory");
          else
            asm volatile(
                "{\n\t.reg .pred p;\n\t"
                "setp.eq.b32 p, 0, 0;\n\t"
                "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
                ::"r"(d_t), "r"(op_t), "l"(bd), "r"(idesc)
                : "memory");
        }
        asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                         BAR_ADDR(done, slot))
                     : "memory");
        ready = next0 && next1;
        slot = slot1; phase = phase1;
      }
    }
  }

  if (p.cluster > 1 && warp < W_EPI) {
    // the tile's sums to the set's hand-over buffer
    __syncwarp();
    asm volatile("griddepcontrol.wait;" ::: "memory");  // C may still be in use by the previous kernel
    float4* hand = reinterpret_cast<float4*>(smem_al + hand_off + (uint32_t)(warp >> 2) * HAND) + (warp & 3) * 32 + lane;
#pragma unroll
    for (int q = 0; q < 4; ++q)
      if (q * 4 < p.M) hand[q * 128] = make_float4(acc[4 * q], acc[4 * q + 1], acc[4 * q + 2], acc[4 * q + 3]);
  }

  // ================= teardown =================
  __syncwarp();
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (*abort_flag && tid == 0) {
    atomicExch(p.status, ST_DEVICE_TIMEOUT);
    p.status[1] = 10;  // where: exact small-batch kernel pipeline
    p.status[2] = blockIdx.x;
    p.status[3] = 0;
  }
  if (warp == W_MMA) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem) : "memory");
  }
  if (p.cluster > 1) {
    cluster_arrive();
    cluster_wait();
    if (warp < W_EPI && !*abort_flag)
      cluster_finish<ACT, EXACT_SETS>(p, smem_base + hand_off, HAND, blockIdx.x % p.cluster, run0 / p.G, (warp & 3) * 32 + lane, lane,
                          warp >> 2, EXACT_SETS);
    cluster_arrive();  // nobody leaves while its sums are being read
    cluster_wait();
  }
#undef BAR_ADDR
}

template <int VAR, int ACT>
static cudaError_t exact_launch_one(const BatchParams& p, const CUtensorMap* tmaps, int smem_bytes, cudaStream_t stream) {
  auto kern = exact_kernel<VAR, ACT>;
  static std::atomic<bool> allowed[16];
  const cudaError_t e = allow_smem(kern, allowed);
  if (e != cudaSuccess) return e;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)p.grid, 1, 1);
  cfg.blockDim = dim3(EXACT_THREADS, 1, 1);
  cfg.dynamicSmemBytes = (size_t)smem_bytes;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = (unsigned)p.cluster;
  attr[1].val.clusterDim.y = 1;
  attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = p.cluster > 1 ? 2 : 1;
  return cudaLaunchKernelEx(&cfg, kern, p, tmaps[0], tmaps[1]);
}

template <int VAR>
static cudaError_t exact_launch_var(int var, const BatchParams& p, const CUtensorMap* tmaps, int smem_bytes,
                                    cudaStream_t stream) {
  if constexpr (VAR % B200Q_NPARTS == B200Q_PART) {
    if (var == VAR)
      return p.act == 0 ? exact_launch_one<VAR, 0>(p, tmaps, smem_bytes, stream)
                        : exact_launch_one<VAR, 1>(p, tmaps, smem_bytes, stream);
  }
  if constexpr (VAR + 1 < VAR_COUNT) return exact_launch_var<VAR + 1>(var, p, tmaps, smem_bytes, stream);
  else return cudaErrorInvalidValue;
}

#define B200Q_CAT2(a, b) a##b
#define B200Q_CAT(a, b) B200Q_CAT2(a, b)

// One of these per compiled part; api.cu picks the part as var % B200Q_NPARTS.
cudaError_t B200Q_CAT(exact_launch_part, B200Q_PART)(int var, const BatchParams& p, const void* tmaps, int smem_bytes,
                                                     cudaStream_t stream) {
  return exact_launch_var<0>(var, p, reinterpret_cast<const CUtensorMap*>(tmaps), smem_bytes, stream);
}

#if B200Q_PART == 0
// dynamic shared memory: alignment slack + activation groups + packed ring with scales + handed sums + barriers
int exact_smem_bytes(int bits, int stages, int M) {
  return 1024 + EXACT_SLOTS * (int)EXACT_ASTAGE + stages * batch_stage_bytes(bits, 1) + EXACT_SETS * (int)exact_hand_bytes(M) +
         (int)sizeof(ExactBarriers);
}
// Ring stages (a multiple of the sets).  Up to 8 rows within half an SM's shared memory where that holds two stages per
// set (nine of 4-bit weights); 7 and 8 bits get one there, whose copy and decoding cannot overlap (8 x 8192 x 8192, 8 bits:
// 22.3 us with 3 stages, 20.4 with 9).  The half was meant for a launch that follows on the same SM; the registers
// keep that from happening, so the limit only bounds the ring.
int exact_stages(int bits, int max_smem, int M) {
  const int half = 113 * 1024;
  const int cap = M <= 8 && exact_smem_bytes(bits, 2 * EXACT_SETS, M) <= half ? half : max_smem;
  int st = EXACT_STAGES_MAX;
  while (st > EXACT_SETS && exact_smem_bytes(bits, st, M) > cap) st -= EXACT_SETS;
  return st;
}
#endif

}  // namespace b200q
