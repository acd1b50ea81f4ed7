// Batches of up to 128 rows: C[M, N] = A[M, K] x dequant(Bq[K, N]) on tcgen05, weights streamed once.
//
// The product is computed transposed, D[n, m] = sum_k W[k, n] * A[m, k], like the prefill kernel
// (umma_kernel.cu): the dequantized weights are the tensor-memory operand (128 lanes = 128 columns), the
// activations the shared-memory operand with as many rows as the batch has, rounded up to 16.  An MMA of
// 128 x NR x 16 then costs NR / 2 tensor cycles (9 for 16 rows), so that the tensor pipe stays below the HBM
// time of the weights up to about 80 rows of 4-bit weights, and nothing the weights pass through is
// wider than their packed form: global -> (tiled copy) -> shared -> registers -> tensor memory.
//
// Roles of the warps of a CTA, 16 with two dequantizing sets, 20 with three (api.cu, batch_sets):
//   * the first 8 or 12 dequantize, in sets of four (a set covers the 128 lanes; lane L is column L of the
//     tile).  Set s takes the 128-row groups s, s + sets, ... of the CTA: a lane reads its column's four
//     units, decodes and scales them (decode.cuh, unit_decode_scaled: the weights the reference
//     multiplies by, examples/quantization/matmul_a16wx.py:316-320) and writes 64 tensor-memory columns.
//     Each set has operand slots and ring stages of its own, so that every waiter of a ring barrier sees each
//     of its phases in turn.  Two sets leave a third of the time to latencies: 620 cycles per group, 416 of them
//     instructions (64 x 16384 x 4096, 4 bits 15.6 us, with three sets 14.6);
//   * the next four warps are the epilogue; the dequantize warps take a share of the run's last segment.  They
//     do not follow the accumulators' barriers (d_full) from segment to segment - with few groups per tile they are
//     several segments ahead of the MMAs, and a phase of two segments ago would pass for the last one's -
//     but wait for a barrier of one phase, run_done, that the last MMA of the run completes;
//   * one warp brings the activations, two 2-D tiled TMA copies (128-byte swizzle) per group;
//   * one warp brings packed weights, a 128-row group of the 128 columns at a time: one 3-D tiled
//     TMA copy for the eight 16-column pieces.  For 2, 4 and 8 bits it swizzles 16-byte chunks by
//     128-byte line, which spreads eight neighbouring columns over all shared-memory banks (columns are
//     16 * b bytes apart: unswizzled, 4-bit loads would collide four ways); other widths are left dense
//     (two-way);
//   * one warp owns tensor memory and issues eight tcgen05.mma per group;
//   * the last warp brings the scales.
// The four single-thread roles run under elect.sync: copies and MMAs take their operands from uniform
// registers.  (Eight lanes issuing one 1 KB bulk copy each took 1100 cycles per group; the copies of a
// group may take 360 at the HBM rate of 4-bit weights.)
//
// Work split.  The (column tile, 128-row group) pairs are numbered tile by tile and cut into equal
// contiguous runs, one per CTA, whatever the shape.  A run covers at most one tile's end, whole
// tiles, and one tile's start.  Whole tiles are written to C; a partial tile's sums are added into an
// fp32 scratch tile (red.global.add.v4) and counted in, and whoever completes the count converts them,
// writes C and puts the scratch back to zero (batch_epilogue).  These additions are the price of the form:
// 4.8 MB of them at 64 rows keep L2 busy for 6 us.  Where the column tiles are few enough that every one can have
// a cluster of CTAs to itself, the launch takes the cluster form instead, whose CTAs send their sums to one another in bulk
// copies (cluster_epilogue); where they fill one round of SMs, whole column tiles (the rule is in api.cu).
//
// Measured (4-bit, group 128, a chain of cold launches; the kernel before it wrote dequantized weights to
// 256-column shared-memory operands): 64 x 28672 x 4096 44.5 -> 24.9 us, 64 x 8192 x 8192 28.2 -> 17.1,
// 128 x 8192 x 8192 34.0 -> 19.2.  What is left at 64 rows is the dequantize warps' instructions and
// the additions of the partial tiles in L2.
//
// Every mbarrier wait is bounded in time; a wait that runs out raises a CTA-wide abort flag, all loops
// leave, the producers give their copies in flight a bounded chance to land, tensor memory is freed and
// the status word of the workspace reports it.
#include <cuda.h>

#include "common.cuh"
#include "batch_common.cuh"

#ifndef B200Q_PART
#define B200Q_PART 0
#endif
#ifndef B200Q_NPARTS
#define B200Q_NPARTS 1
#endif

namespace b200q {

constexpr int batch_threads(int sets) { return sets * 128 + 256; }  // + four epilogue warps, three producers, MMA warp
constexpr int BATCH_SLOTS_MAX = 6;                 // 128-row operand slots, of 64 tensor-memory columns
constexpr int BATCH_STAGES_MAX = 16;               // 128-row groups in the packed ring, a multiple of the sets
constexpr int BATCH_A_MAX = 6;                     // 128-row activation groups in shared memory, at most the slots

struct BatchBarriers {
  uint64_t slot_full[BATCH_SLOTS_MAX];
  uint64_t done[BATCH_SLOTS_MAX];  // [i]: the MMAs of a group in slot i have completed
  uint64_t a_full[BATCH_A_MAX];
  uint64_t g_full[BATCH_STAGES_MAX], g_empty[BATCH_STAGES_MAX];
  uint64_t d_full[2], d_empty[2];
  uint64_t run_done;  // the MMAs of the whole run have completed
  uint64_t sums_full[4];  // cluster form, per lane quadrant: all CTAs' sums of this CTA's rows are here
  uint32_t tmem_base;
  volatile int abort_flag;
};
constexpr int BATCH_BARRIERS = (int)(offsetof(BatchBarriers, tmem_base) / 8);
// arrivals that complete a phase of the i-th barrier
__host__ __device__ constexpr int batch_barrier_count(int i, int sets) {
  return i < (int)(offsetof(BatchBarriers, done) / 8) ? 4
       : i < (int)(offsetof(BatchBarriers, g_full) / 8) ? 1
       : i < (int)(offsetof(BatchBarriers, g_empty) / 8) ? 2
       : i < (int)(offsetof(BatchBarriers, d_full) / 8) ? 4
       : i < (int)(offsetof(BatchBarriers, d_empty) / 8) ? 1
       : i < (int)(offsetof(BatchBarriers, run_done) / 8) ? 4
       : i < (int)(offsetof(BatchBarriers, sums_full) / 8) ? 1 : sets + 1;
}

// tensor memory (all 512 columns): two D accumulators of nr columns - one for three sets beyond 64 rows, whose CTAs have a single
// column tile - then the operand slots
__host__ __device__ constexpr int batch_d_stride(int nr) { return nr <= 64 ? 64 : 128; }
__host__ __device__ constexpr int batch_d_count(int nr, int sets) { return sets == 3 && nr > 64 ? 1 : 2; }
__host__ __device__ constexpr int batch_slots(int nr, int sets) { return (512 - batch_d_count(nr, sets) * batch_d_stride(nr)) / 64; }

// The epilogue of one segment, shared out over `parts` groups of four warps (this warp belongs to group
// `part`): rows in chunks of 16 from tensor memory, to C (a whole tile) or added into the tile's scratch.
// Each (lane quadrant, chunk) of a tile is counted by itself, in 128-row groups: the warp that completes
// the count converts its sums, writes C and puts sums and count back to zero.  Nothing waits for the rest of
// the CTA.  (Slabs per CTA with plain stores, added up by the last to arrive, measured slower: its loads of
// lines other SMs have just written cost 2 - 8 us more than these additions.)
template <int ACT>
__device__ __forceinline__ void batch_epilogue(const BatchParams& p, uint32_t d_t, uint32_t d_empty, int tile, int len,
                                               int wq, int lane, int part, int parts) {
  const int nl = wq * 32 + lane, n = tile * 128 + nl;
  const bool whole = len == p.G;
  float4* sums = reinterpret_cast<float4*>(p.partial) + (size_t)tile * (p.rows * 32) + nl;
  for (int c0 = part * 16; c0 < p.M; c0 += 16 * parts) {
    uint32_t v[16];
    tmem_ld_16(d_t + (uint32_t)c0, v);
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int m = c0 + q * 4;
      if (m >= p.M) continue;
      const float4 f = make_float4(__uint_as_float(v[4 * q]), __uint_as_float(v[4 * q + 1]), __uint_as_float(v[4 * q + 2]),
                                   __uint_as_float(v[4 * q + 3]));
      if (whole)
        batch_store4<ACT>(p, n, lane, m, f);
      else
        asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(sums + (m >> 2) * 128), "f"(f.x), "f"(f.y),
                     "f"(f.z), "f"(f.w)
                     : "memory");
    }
  }
  // the accumulator has been read: the MMAs of the segment after next may overwrite it
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncwarp();
  if (d_empty != 0 && lane == 0) mbar_arrive(d_empty);
  if (!whole) batch_finish<ACT>(p, tile, len, wq, lane, part, parts);
}

// The end of a column tile whose K a cluster shares, by the twelve warps that know of tensor memory.  The rows are cut into quads of four,
// of which the CTAs own equal shares (the last ones what is left).  A warp takes 16 rows of its 32 columns at a time from tensor
// memory to the CTA's own shared memory (over the activations: all MMAs have completed), [quad][32] float4, and sends each owner
// its quads with one bulk copy, which counts its bytes in on the owner's barrier of the lane quadrant, as the owner's own warps
// count themselves in.  The owner adds the
// CTAs' sums in rank order and writes C.  A CTA that has all of its sums says so on the cluster's barrier and waits for the others
// before it leaves, since until then its own copies may not have been read.  (64 x 4096 x 4096, three CTAs per tile, us per launch: sums
// left in place and fetched by their owners between two barriers of the cluster 9.8, the last 3 of them; sent word by word 9.2.)
__host__ __device__ constexpr int batch_own_quads(int quads, int cluster) { return (quads + cluster - 1) / cluster; }
template <int ACT, int SETS>
__device__ __forceinline__ void cluster_epilogue(const BatchParams& p, uint32_t tmem, const unsigned char* smem, uint32_t smem_s,
                                                 uint32_t sums_off, uint32_t run_done, uint32_t full, int tile, int warp, int lane,
                                                 volatile int* abort_flag) {
  const int wq = warp & 3, part = warp >> 2, rank = blockIdx.x % p.cluster;
  const int quads = (p.M + 3) / 4, own = batch_own_quads(quads, p.cluster);
  const int q0 = min(quads, rank * own), q1 = min(quads, q0 + own);  // this CTA's
  const uint32_t sent = smem_s + (uint32_t)(wq * quads) * 512u;
  const uint32_t got_off = sums_off + (uint32_t)(wq * (p.cluster - 1) * own) * 512u;  // [other CTA][owned quad][32]
  bool ok = mbar_wait_abortable(run_done, 0u, abort_flag);
  if (__all_sync(0xffffffffu, ok ? 1 : 0)) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    for (int c0 = part * 4; c0 < quads; c0 += 4 * (SETS + 1)) {
      uint32_t v[16];
      tmem_ld_16(tmem + ((uint32_t)(wq * 32) << 16) + (uint32_t)(c0 * 4), v);
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (c0 + u < quads)
          asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(sent + (uint32_t)((c0 + u) * 512 + lane * 16)), "r"(v[4 * u]),
                       "r"(v[4 * u + 1]), "r"(v[4 * u + 2]), "r"(v[4 * u + 3])
                       : "memory");
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncwarp();
    if (elect_one()) {
      if (part == 0)
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(full), "r"((uint32_t)((q1 - q0) * (p.cluster - 1)) * 512u)
                     : "memory");
      else
        mbar_arrive(full);
      for (int c0 = part * 4; c0 < quads; c0 += 4 * (SETS + 1)) {
        const int c1 = min(quads, c0 + 4);
        for (int q = c0, owner = c0 / own; q < c1; ++owner) {
          const int next = min(c1, (owner + 1) * own), place = rank - (rank > owner ? 1 : 0);
          if (owner == rank) { q = next; continue; }
          uint32_t dst, bar;
          asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(dst)
                       : "r"(smem_s + got_off + (uint32_t)(place * own + q - owner * own) * 512u), "r"(owner));
          asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(bar) : "r"(full), "r"(owner));
          asm volatile("cp.async.bulk.shared::cluster.shared::cta.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
                       "r"(sent + (uint32_t)q * 512u), "r"((uint32_t)(next - q) * 512u), "r"(bar)
                       : "memory");
          q = next;
        }
      }
    }
    __syncwarp();
    ok = mbar_wait_abortable(full, 0u, abort_flag);
    ok = __all_sync(0xffffffffu, ok ? 1 : 0);
  } else {
    ok = false;
  }
  cluster_arrive_relaxed();
  if (!ok) return;
  const float4* parts = reinterpret_cast<const float4*>(smem + got_off) + lane;
  const float4* mine = reinterpret_cast<const float4*>(smem) + (wq * quads + q0) * 32 + lane;
#pragma unroll 2
  for (int q = part; q < q1 - q0; q += SETS + 1) {
    float4 sum = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 4
    for (int r = 0; r < p.cluster; ++r) {
      const float4 x = r == rank ? mine[q * 32] : parts[((r - (r > rank ? 1 : 0)) * own + q) * 32];
      sum.x += x.x; sum.y += x.y; sum.z += x.z; sum.w += x.w;
    }
    batch_store4<ACT>(p, tile * 128 + wq * 32 + lane, lane, (q0 + q) * 4, sum);
  }
}

template <int VAR, int ACT, bool CLUSTER, int SETS>
__device__ __forceinline__ void batch_body(const BatchParams& p, const CUtensorMap& tmap_a, const CUtensorMap& tmap_w) {
  constexpr int B = var_bits(VAR);
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  const uint32_t smem_unaligned = (uint32_t)__cvta_generic_to_shared(smem_raw);
  const uint32_t smem_base = (smem_unaligned + 1023u) & ~1023u;
  unsigned char* smem_al = smem_raw + (smem_base - smem_unaligned);
  const int NR = p.rows, WS = p.stages, AS = p.a_stages;
  constexpr uint32_t WSTAGE = 2048u * B;
  const uint32_t ASTAGE = (uint32_t)NR * 256u, SSTAGE = 256u * (uint32_t)p.rpg;
  const uint32_t ring_off = (uint32_t)AS * ASTAGE, scales_off = ring_off + (uint32_t)WS * WSTAGE;
  const uint32_t ring_s = smem_base + ring_off, scales_s = smem_base + scales_off;
  const uint32_t bars_off = scales_off + (uint32_t)WS * SSTAGE;
  const uint32_t sums_off = bars_off + (uint32_t)((sizeof(BatchBarriers) + 127) / 128 * 128);  // what a cluster's CTAs send
  BatchBarriers* bars = reinterpret_cast<BatchBarriers*>(smem_al + bars_off);
  const uint32_t bars_s = smem_base + bars_off;
#define BAR_ADDR(field, i) (bars_s + (uint32_t)offsetof(BatchBarriers, field) + (uint32_t)(i) * 8u)

  const int tid = threadIdx.x, lane = tid & 31;
  const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
  volatile int* abort_flag = &bars->abort_flag;
  // this CTA's run of groups, counted tile by tile over the whole matrix
  const int run0 = batch_run_start(p, blockIdx.x), run1 = batch_run_start(p, blockIdx.x + 1);

  constexpr int TM_THREADS = SETS * 128 + 160;
  constexpr int W_EPI = SETS * 4, W_ACT = W_EPI + 4, W_WEIGHTS = W_EPI + 5, W_MMA = W_EPI + 6,
                W_SCALES = W_EPI + 7;
  // (The descriptors are on their way while the barriers are set up, by the lanes of one warp.  Thread 0 alone took 1800 cycles
  // for both, ahead of the first copies.)
  if (warp == W_WEIGHTS && lane == 0) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(&tmap_w) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&tmap_a) : "memory");
  }
  if (warp == 0) {
    for (int i = lane; i < BATCH_BARRIERS; i += 32) mbar_init(bars_s + (uint32_t)i * 8u, (uint32_t)batch_barrier_count(i, SETS));
    if (lane == 0) bars->abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  __syncthreads();
  if constexpr (CLUSTER) {  // (the peers' barriers are there before anything is sent to them)
    cluster_arrive();
    cluster_wait();
  }
  // the producers may start; the roles that use tensor memory wait for it below (the previous launch's CTA on
  // this SM may still hold it)
  if (warp == W_MMA) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(
                     bars_s + (uint32_t)offsetof(BatchBarriers, tmem_base))
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    // Only now may the next launch start: a CTA of it that got this SM's tensor memory first would wait for this
    // launch to complete, and this launch for the tensor memory.  (With this order a launch whose CTAs wait for
    // their predecessor never holds tensor memory that the predecessor still has to get, on whatever streams.)
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  }
  if (warp < W_ACT || warp == W_MMA) {
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    asm volatile("bar.sync 1, %0;" ::"n"(TM_THREADS) : "memory");
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  }
  const uint32_t tmem = (warp < W_ACT || warp == W_MMA) ? __shfl_sync(0xffffffffu, bars->tmem_base, 0) : 0u;
  const int nslots = batch_slots(NR, SETS), n_d = batch_d_count(NR, SETS), d_stride = batch_d_stride(NR);
  const uint32_t slots_t = tmem + (uint32_t)(n_d * d_stride);

  // one segment of the run: pos -> tile, groups
#define SEGMENT(pos)                                     \
  const int tile = (pos) / p.G, g0 = (pos) - tile * p.G; \
  const int len = min(p.G - g0, run1 - (pos));           \
  const bool last_seg = (pos) + len == run1;             \
  (void)last_seg;

  if (warp < W_EPI) {
    // ================= dequantize (and a share of the last segment's epilogue) =================
    const int set = warp >> 2, wq = warp & 3;
    const int nl = wq * 32 + lane;  // lane of tensor memory = column inside the tile
    const uint32_t lane_t = (uint32_t)(wq * 32) << 16;
    bool good = true;
    int stage = set, slot = set;    // stages of a set: set, set + SETS, ...; slots likewise
    uint32_t ring_phase = 0, slot_phase = 1;
    for (int g_own = set; g_own < run1 - run0; g_own += SETS) {
      if (!mbar_wait_abortable(BAR_ADDR(g_full, stage), ring_phase, abort_flag)) { good = false; break; }
      const uint32_t st = ring_s + (uint32_t)stage * WSTAGE;
      const uint32_t sc = scales_s + (uint32_t)stage * SSTAGE + (uint32_t)nl * 2u;
      uint32_t w[2][2 * B], s2[4];
      unsigned short sb;
      asm volatile("ld.shared.u16 %0, [%1];" : "=h"(sb) : "r"(sc));
      s2[0] = s2[1] = s2[2] = s2[3] = (uint32_t)sb * 0x00010001u;  // the 16-bit scale in both halves
      if (p.rpg > 1) {
#pragma unroll
        for (int u = 1; u < 4; ++u) {
          asm volatile("ld.shared.u16 %0, [%1];" : "=h"(sb) : "r"(sc + (uint32_t)((u * p.rpg) >> 2) * 256u));
          s2[u] = (uint32_t)sb * 0x00010001u;
        }
      }
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        batch_load_units<B>(st, nl, h, w[h]);
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          uint32_t out[16];
          unit_decode_scaled<VAR, ACT>(w[h] + u * B, s2[2 * h + u], out);
          if (h == 0 && u == 0) {  // the MMAs have read what the set stored here before
            if (!mbar_wait_abortable(BAR_ADDR(done, slot), slot_phase, abort_flag)) { good = false; break; }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          }
          if (h == 1 && u == 0) {  // the stage has been read (its values fed the arithmetic above)
            __syncwarp();
            if (lane == 0) mbar_arrive(BAR_ADDR(g_empty, stage));
          }
          tmem_st_16(slots_t + lane_t + (uint32_t)(slot * 64 + h * 32 + u * 16), out);
        }
        if (!good) break;
      }
      if (!good) break;
      asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(BAR_ADDR(slot_full, slot));
      slot += SETS;
      if (slot >= nslots) { slot = set; slot_phase ^= 1u; }
      stage += SETS;
      if (stage >= WS) { stage = set; ring_phase ^= 1u; }
    }
    if (!CLUSTER && good) {
      int pos = run0, seg = 0;  // the last segment
      while (pos / p.G != (run1 - 1) / p.G) { pos = (pos / p.G + 1) * p.G; ++seg; }
      SEGMENT(pos)
      asm volatile("griddepcontrol.wait;" ::: "memory");  // C and the scratch may still be in use by the previous kernel
      if (mbar_wait_abortable(BAR_ADDR(run_done, 0), 0u, abort_flag)) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        batch_epilogue<ACT>(p, tmem + lane_t + (uint32_t)((seg % n_d) * d_stride), 0u, tile, len, wq, lane, set,
                            SETS + 1);
      }
    }
  } else if (warp < W_ACT) {
    // ================= epilogue =================
    const int wq = warp & 3;
    const uint32_t lane_t = (uint32_t)(wq * 32) << 16;
    asm volatile("griddepcontrol.wait;" ::: "memory");  // C and the scratch may still be in use by the previous kernel
    int seg = 0;
    for (int pos = run0; pos < run1 && !CLUSTER; ++seg) {
      SEGMENT(pos)
      if (!mbar_wait_abortable(BAR_ADDR(d_full, seg % n_d), (uint32_t)(seg / n_d) & 1u, abort_flag)) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      batch_epilogue<ACT>(p, tmem + lane_t + (uint32_t)((seg % n_d) * d_stride), BAR_ADDR(d_empty, seg % n_d), tile,
                          len, wq, lane, last_seg ? SETS : 0, last_seg ? SETS + 1 : 1);
      pos += len;
    }
  } else if (warp == W_ACT) {
    // ================= TMA producer: activations =================
    if (elect_one()) {
      asm volatile("griddepcontrol.wait;" ::: "memory");
      // The ring's stage of group i held group i - AS, whose MMAs report on its slot's barrier: one commit per
      // group frees slot and activations (a second commit right behind the first costs the issuing thread
      // 600 cycles).
      int stage = 0, n_issued = 0, slot = 0;
      uint32_t phase = 0;
      bool good = true;
      int g = run0 % p.G;
      for (int pos = run0; pos < run1; ++pos) {
        if (n_issued >= AS) {
          if (!mbar_wait_abortable(BAR_ADDR(done, slot), phase, abort_flag)) { good = false; break; }
          if (++slot == nslots) { slot = 0; phase ^= 1u; }
        }
        const uint32_t bar = BAR_ADDR(a_full, stage);
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(ASTAGE) : "memory");
#pragma unroll
        for (int h = 0; h < 2; ++h)
          asm volatile(
              "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
              ::"r"(smem_base + (uint32_t)stage * ASTAGE + (uint32_t)h * (ASTAGE / 2)), "l"(&tmap_a), "r"(bar),
              "r"(g * 128 + h * 64), "r"(0)
              : "memory");
        ++n_issued;
        if (++stage == AS) stage = 0;
        if (++g == p.G) g = 0;
      }
      if (!good) {  // a copy in flight must not outlive the CTA: a bounded wait for the groups issued last
        for (int i = max(0, n_issued - AS); i < n_issued; ++i)
          mbar_wait_bounded(BAR_ADDR(a_full, i % AS), (uint32_t)(i / AS) & 1u);
      }
    }
  } else if (warp == W_WEIGHTS) {
    // ================= TMA producer: packed weights =================
    if (elect_one()) {
      int stage = 0, n_issued = 0;
      uint32_t phase = 1;
      bool good = true;
      int tile = run0 / p.G, g = run0 - tile * p.G;
      for (int pos = run0; pos < run1; ++pos) {
        if (!mbar_wait_abortable(BAR_ADDR(g_empty, stage), phase, abort_flag)) { good = false; break; }
        const uint32_t bar = BAR_ADDR(g_full, stage);
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(WSTAGE) : "memory");
        // (pieces past the last column are filled with zeros and count as bytes all the same)
        asm volatile(
            "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
            ::"r"(ring_s + (uint32_t)stage * WSTAGE), "l"(&tmap_w), "r"(bar), "r"(0),
            "r"(batch_swizzled(B) ? g * (2 * B) : g), "r"(tile * 8)
            : "memory");
        ++n_issued;
        if (++g == p.G) { g = 0; ++tile; }
        if (++stage == WS) { stage = 0; phase ^= 1u; }
      }
      if (!good) {
        for (int i = max(0, n_issued - WS); i < n_issued; ++i)
          mbar_wait_bounded(BAR_ADDR(g_full, i % WS), (uint32_t)(i / WS) & 1u);
      }
    }
  } else if (warp == W_SCALES) {
    // ================= bulk-copy producer: scales (a thread of its own: issuing takes 100 cycles a copy) =================
    if (elect_one()) {
      int stage = 0, n_issued = 0;
      uint32_t phase = 1;
      bool good = true;
      int tile = run0 / p.G, g = run0 - tile * p.G;
      // scale row(s) of the group: p.rpg rows per group, or one row for p.group / 128 groups
      const int groups_per_row = p.rpg == 1 ? p.group / 128 : 1;
      int in_row = g % groups_per_row;
      const __half* sc = p.scales + (size_t)(p.rpg == 1 ? g / groups_per_row : g * p.rpg) * p.N + tile * 128;
      uint32_t sc_bytes = (uint32_t)min(128, p.N - tile * 128) * 2u;
      for (int pos = run0; pos < run1; ++pos) {
        if (!mbar_wait_abortable(BAR_ADDR(g_empty, stage), phase, abort_flag)) { good = false; break; }
        const uint32_t bar = BAR_ADDR(g_full, stage);
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(sc_bytes * (uint32_t)p.rpg)
                     : "memory");
        for (int i = 0; i < p.rpg; ++i)
          asm volatile(
              "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                  scales_s + (uint32_t)stage * SSTAGE + (uint32_t)i * 256u),
              "l"(sc + (size_t)i * p.N), "r"(sc_bytes), "r"(bar)
              : "memory");
        ++n_issued;
        if (++in_row == groups_per_row) { in_row = 0; sc += (size_t)p.rpg * p.N; }
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
      const uint32_t idesc = umma_idesc<ACT>(NR);
      bool good = true;
      int slot = 0, stage = 0, seg = 0;
      uint32_t slot_phase = 0, a_phase = 0;
      // the next group's barriers are looked at before this group's MMAs are issued, so that the latency of
      // the look (twice 100 cycles) lies under them; only a group that was not ready then is waited for
      bool ready = false;
      for (int pos = run0; pos < run1 && good; ++seg) {
        SEGMENT(pos)
        if (!mbar_wait_abortable(BAR_ADDR(d_empty, seg % n_d), ((uint32_t)(seg / n_d) & 1u) ^ 1u, abort_flag)) { good = false; break; }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t d_t = tmem + (uint32_t)((seg % n_d) * d_stride);
        for (int i = 0; i < len && good; ++i) {
          if (!ready && (!mbar_wait_abortable(BAR_ADDR(slot_full, slot), slot_phase, abort_flag) ||
                         !mbar_wait_abortable(BAR_ADDR(a_full, stage), a_phase, abort_flag))) { good = false; break; }
          const int slot1 = slot + 1 == nslots ? 0 : slot + 1, stage1 = stage + 1 == AS ? 0 : stage + 1;
          const uint32_t slot_phase1 = slot_phase ^ (slot1 == 0 ? 1u : 0u), a_phase1 = a_phase ^ (stage1 == 0 ? 1u : 0u);
          const bool next0 = mbar_test(BAR_ADDR(slot_full, slot1), slot_phase1);
          const bool next1 = mbar_test(BAR_ADDR(a_full, stage1), a_phase1);
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const uint64_t bdesc = umma_smem_desc(smem_base + (uint32_t)stage * ASTAGE);
          const uint32_t a_t = slots_t + (uint32_t)(slot * 64), half = ASTAGE >> 5;  // second block, in 16-byte units
#pragma unroll
          for (int ks = 0; ks < 8; ++ks) {
            const uint32_t accumulate = (i > 0 || ks > 0) ? 1u : 0u;
            asm volatile(
                "{\n\t.reg .pred p;\n\t"
                "setp.ne.b32 p, %4, 0;\n\t"
                "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
                ::"r"(d_t), "r"(a_t + (uint32_t)(ks * 8)), "l"(bdesc + (uint64_t)((ks & 3) * 2) + (ks < 4 ? 0u : half)),
                "r"(idesc), "r"(accumulate)
                : "memory");
          }
          asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                           BAR_ADDR(done, slot))
                       : "memory");
          ready = next0 && next1;
          slot = slot1; slot_phase = slot_phase1; stage = stage1; a_phase = a_phase1;
        }
        if (good)
          asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                           BAR_ADDR(d_full, seg % n_d))
                       : "memory");
        pos += len;
      }
      if (good)
        asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                         BAR_ADDR(run_done, 0))
                     : "memory");
    }
  }

  if constexpr (CLUSTER) {
    __syncwarp();
    if (warp < W_ACT) {
      asm volatile("griddepcontrol.wait;" ::: "memory");  // C may still be in use by the previous kernel
      cluster_epilogue<ACT, SETS>(p, tmem, smem_al, smem_base, sums_off, BAR_ADDR(run_done, 0), BAR_ADDR(sums_full, warp & 3), run0 / p.G,
                            warp, lane, abort_flag);
    } else {
      cluster_arrive_relaxed();
    }
  }

  // ================= teardown =================
  __syncwarp();
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (*abort_flag && tid == 0) {
    atomicExch(p.status, ST_DEVICE_TIMEOUT);
    p.status[1] = 6;  // where: small-batch tcgen05 kernel pipeline
    p.status[2] = blockIdx.x;
    p.status[3] = 0;
  }
  if (warp == W_MMA) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem) : "memory");
  }
  if constexpr (CLUSTER) cluster_wait();  // everybody has what was sent from here, and nothing more is on its way here
#undef BAR_ADDR
#undef SEGMENT
}

// Equal runs with two sets: of up to 32 rows, of which two CTAs have registers on an SM (64, see batch_stages), and of more than 64.
// Equal runs with three sets, and a cluster of CTAs per column tile (api.cu, batch_sets).
// (float4, and 7-bit integers in bfloat16, would take 69 to 72 registers and do with 64 without spills; the others' code is slower for
// being told.)
constexpr bool batch_told_registers(int var, int act) { return var == VAR_F4E2M1 || (!var_is_float(var) && var_bits(var) == 7 && act == 1); }
template <int VAR, int ACT>
__global__ void __launch_bounds__(batch_threads(2), batch_told_registers(VAR, ACT) ? 2 : 1)
batch_kernel(const __grid_constant__ BatchParams p, const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_w) {
  batch_body<VAR, ACT, false, 2>(p, tmap_a, tmap_w);
}
template <int VAR, int ACT>
__global__ void __launch_bounds__(batch_threads(3), 1)
tile_run_kernel(const __grid_constant__ BatchParams p, const __grid_constant__ CUtensorMap tmap_a,
                const __grid_constant__ CUtensorMap tmap_w) {
  batch_body<VAR, ACT, false, 3>(p, tmap_a, tmap_w);
}
template <int VAR, int ACT, int SETS>
__global__ void __launch_bounds__(batch_threads(SETS), 1)
tile_cluster_kernel(const __grid_constant__ BatchParams p, const __grid_constant__ CUtensorMap tmap_a,
                    const __grid_constant__ CUtensorMap tmap_w) {
  batch_body<VAR, ACT, true, SETS>(p, tmap_a, tmap_w);
}

template <int VAR, int ACT, bool CLUSTER, int SETS>
static cudaError_t batch_launch_one(const BatchParams& p, const CUtensorMap* tmaps, int smem_bytes, cudaStream_t stream) {
  auto kern = CLUSTER ? tile_cluster_kernel<VAR, ACT, SETS> : SETS == 3 ? tile_run_kernel<VAR, ACT> : batch_kernel<VAR, ACT>;
  static std::atomic<bool> allowed[16];
  const cudaError_t e = allow_smem(kern, allowed);
  if (e != cudaSuccess) return e;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)p.grid, 1, 1);
  cfg.blockDim = dim3((unsigned)batch_threads(SETS), 1, 1);
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

template <int VAR, bool CLUSTER, int SETS>
static cudaError_t batch_launch_act(const BatchParams& p, const CUtensorMap* tmaps, int smem_bytes, cudaStream_t stream) {
  return p.act == 0 ? batch_launch_one<VAR, 0, CLUSTER, SETS>(p, tmaps, smem_bytes, stream)
                    : batch_launch_one<VAR, 1, CLUSTER, SETS>(p, tmaps, smem_bytes, stream);
}

template <int VAR>
static cudaError_t batch_launch_var(int var, const BatchParams& p, const CUtensorMap* tmaps, int smem_bytes,
                                    cudaStream_t stream) {
  if constexpr (VAR % B200Q_NPARTS == B200Q_PART) {
    if (var == VAR) {
      if (p.cluster > 1)
        return p.sets == 3 ? batch_launch_act<VAR, true, 3>(p, tmaps, smem_bytes, stream) : batch_launch_act<VAR, true, 2>(p, tmaps, smem_bytes, stream);
      return p.sets == 3 ? batch_launch_act<VAR, false, 3>(p, tmaps, smem_bytes, stream) : batch_launch_act<VAR, false, 2>(p, tmaps, smem_bytes, stream);
    }
  }
  if constexpr (VAR + 1 < VAR_COUNT) return batch_launch_var<VAR + 1>(var, p, tmaps, smem_bytes, stream);
  else return cudaErrorInvalidValue;
}

#define B200Q_CAT2(a, b) a##b
#define B200Q_CAT(a, b) B200Q_CAT2(a, b)

// One of these per compiled part; api.cu picks the part as var % B200Q_NPARTS.
cudaError_t B200Q_CAT(batch_launch_part, B200Q_PART)(int var, const BatchParams& p, const void* tmaps, int smem_bytes,
                                                     cudaStream_t stream) {
  return batch_launch_var<0>(var, p, reinterpret_cast<const CUtensorMap*>(tmaps), smem_bytes, stream);
}

#if B200Q_PART == 0
// clusters of c CTAs that the current device holds at a time with one CTA per SM; 0 without a device
int batch_max_clusters(int c) {
  auto kern = tile_cluster_kernel<0, 0, 3>;
  const int smem = 200 * 1024;
  static std::atomic<bool> allowed[16];
  if (allow_smem(kern, allowed) != cudaSuccess) { (void)cudaGetLastError(); return 0; }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)c, 1, 1);
  cfg.blockDim = dim3((unsigned)batch_threads(3), 1, 1);
  cfg.dynamicSmemBytes = (size_t)smem;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)c;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  int n = 0;
  if (cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess) { (void)cudaGetLastError(); return 0; }
  return n;
}
// dynamic shared memory: alignment slack + activation groups + packed ring + scales + barriers + what a cluster's CTAs send
int batch_smem_bytes(int bits, int stages, int a_stages, int rows, int rpg, int cluster) {
  return 1024 + a_stages * rows * 256 + stages * batch_stage_bytes(bits, rpg) + (int)sizeof(BatchBarriers) +
         (cluster > 1 ? 128 + batch_own_quads(rows / 4, cluster) * (cluster - 1) * 2048 : 0);
}
// Activation groups (at most as many as there are operand slots) and ring stages (a multiple of the dequantize
// sets) in the rest.  Up to 32 rows of 1-, 2- and 4-bit integers and float4 (batch_shares_sm: two sets) a CTA stays within half an SM's
// shared memory and 64 registers, so that the next launch of the stream becomes resident beside this one and fills its ring while
// this one ends (a Llama-3-8B block of linears, 4 bits, at 32 rows: 51 us, 56 with one CTA per SM).  The other types gain more from three sets
// and an SM's whole shared memory (the block at 32 rows, us, so / sharing: 8 bits 57 / 82, whose ring had two stages in a half; 6 bits 59 /
// 61, 3 bits 59 / 60, float6 62 / 66), and more rows leave too little for the ring; launches that leave SMs free (clusters, one CTA per
// column tile) would meet others two to an SM, where one waits for the other's tensor memory (64 rows: 81 us with the two kinds
// mixed, 62).
void batch_stages(int bits, int max_smem, int rows, int rpg, int cluster, int sets, int* stages, int* a_stages) {
  const int cap = rows <= 32 && sets == 2 ? 113 * 1024 : max_smem;
  *a_stages = rows <= 64 ? 6 : 4;
  int st = 0;
  for (;; --*a_stages) {  // (wide types in clusters of many rows: activations make room for a ring of two stages per set)
    st = BATCH_STAGES_MAX / sets * sets;
    while (st > sets && batch_smem_bytes(bits, st, *a_stages, rows, rpg, cluster) > cap) st -= sets;
    if (cluster <= 1 || *a_stages == 2 || (st >= 2 * sets && batch_smem_bytes(bits, st, *a_stages, rows, rpg, cluster) <= cap)) break;
  }
  *stages = st;
}
#endif

}  // namespace b200q
