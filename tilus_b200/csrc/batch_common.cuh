// What the two kernels for small batches share (batch_kernel.cu, exact_kernel.cu): ring stages of packed weights,
// the split of the work over CTAs, and the end of a column tile whose sums come from several CTAs.
#pragma once
#include "umma_common.cuh"

namespace b200q {

// a ring stage: 128 columns x 128 rows of packed weights, and (in a region of their own) rpg rows of 128 scales
__host__ __device__ constexpr int batch_stage_bytes(int bits, int rpg) { return 2048 * bits + 256 * rpg; }
// widths whose stages are swizzled by 128-byte line (see above)
__host__ __device__ constexpr bool batch_swizzled(int bits) { return bits == 2 || bits == 4 || bits == 8; }
// 16 registers -> 16 consecutive tensor-memory columns of this thread's lane
__device__ __forceinline__ void tmem_st_16(uint32_t taddr, const uint32_t (&o)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, "
      "%14, %15, %16};" ::"r"(taddr),
      "r"(o[0]), "r"(o[1]), "r"(o[2]), "r"(o[3]), "r"(o[4]), "r"(o[5]), "r"(o[6]), "r"(o[7]), "r"(o[8]), "r"(o[9]),
      "r"(o[10]), "r"(o[11]), "r"(o[12]), "r"(o[13]), "r"(o[14]), "r"(o[15])
      : "memory");
}

// Four rows (m .. m + 3) of one column per lane -> each lane stores four consecutive columns of one row.
template <int ACT>
__device__ __forceinline__ void batch_store4(const BatchParams& p, int n, int lane, int m, const float4& v) {
  const bool b0 = lane & 1, b1 = lane & 2;
  // two 16-bit rows per register, then two exchange rounds
  const uint32_t r01 = pack2<ACT>(v.x, v.y), r23 = pack2<ACT>(v.z, v.w);
  // round 1 (columns n and n ^ 1): even lane keeps rows 0 and 2, odd lane rows 1 and 3
  const uint32_t o01 = __shfl_xor_sync(0xffffffffu, r01, 1), o23 = __shfl_xor_sync(0xffffffffu, r23, 1);
  const uint32_t x0 = b0 ? __byte_perm(o01, r01, 0x7632) : __byte_perm(r01, o01, 0x5410);  // row 0 + b0
  const uint32_t x2 = b0 ? __byte_perm(o23, r23, 0x7632) : __byte_perm(r23, o23, 0x5410);  // row 2 + b0
  // round 2 (column pairs): lanes with b1 = 0 take row b0, those with b1 = 1 row 2 + b0
  const uint32_t got = __shfl_xor_sync(0xffffffffu, b1 ? x0 : x2, 2);
  const uint2 o = b1 ? make_uint2(got, x2) : make_uint2(x0, got);
  const int row = m + (b1 ? 2 : 0) + (b0 ? 1 : 0);
  if (row < p.M && n < p.N)
    *reinterpret_cast<uint2*>(reinterpret_cast<unsigned short*>(p.c) + (size_t)row * p.ldc + (n & ~3)) = o;
}

// The 2 * B words of units 2h and 2h + 1 of column `nl` from a ring stage.
template <int B>
__device__ __forceinline__ void batch_load_units(uint32_t stage, int nl, int h, uint32_t* w) {
  const uint32_t off = (uint32_t)((nl >> 4) * (256 * B) + (nl & 15) * (16 * B) + h * (8 * B));
  if constexpr (batch_swizzled(B)) {
    const uint32_t line = off >> 7;
#pragma unroll
    for (int q = 0; q < B / 2; ++q) {
      const uint32_t chunk = ((off >> 4) + (uint32_t)q) & 7u;  // a block's chunks lie in one line
      const uint4 v = lds_u4(stage + (line << 7) + ((chunk ^ (line & 7u)) << 4));
      w[4 * q] = v.x; w[4 * q + 1] = v.y; w[4 * q + 2] = v.z; w[4 * q + 3] = v.w;
    }
  } else {
    uint32_t two[2 * B];
    lds_two_units<B>(stage + off, two);
#pragma unroll
    for (int q = 0; q < 2 * B; ++q) w[q] = two[q];
  }
}

// first group of CTA c's run
__device__ __forceinline__ int batch_run_start(const BatchParams& p, int c) {
  if (p.cluster > 1) return (c / p.cluster) * p.G + (c % p.cluster) * p.G / p.cluster;
  return (int)((long long)p.work * c / p.grid) * p.unit;
}

// ---- column tiles shared by the CTAs of a cluster ------------------------------------------------
// Cluster form of a launch (p.cluster > 1): a cluster owns one column tile, its CTAs equal ranges of K.  Every CTA
// leaves its sums in its own shared memory, [quad of four rows][128 columns] float4, and gives its tensor
// memory back BEFORE it waits for the others (another CTA of the cluster may share the SM and wait for that
// memory).  The rows are cut into quads of four; CTA o adds up the quads [Q * o / c, Q * (o + 1) / c) of all
// CTAs in rank order and writes C.
__device__ __forceinline__ void cluster_arrive() {  // orders shared memory accesses before it
  __syncwarp();
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
}
__device__ __forceinline__ void cluster_arrive_relaxed() {  // orders nothing
  __syncwarp();
  asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");
}
__device__ __forceinline__ void cluster_wait() {
  __syncwarp();
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ float4 cluster_load4(uint32_t smem_addr, int rank) {
  uint32_t remote;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(smem_addr), "r"(rank));
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(remote) : "memory");
  return v;
}
// This CTA's quads, dealt over `parts` groups of four warps.  The sums of CTA r lie at sums_s (the same address
// in every CTA), SETS of them set_bytes apart.
template <int ACT, int SETS>
__device__ __forceinline__ void cluster_finish(const BatchParams& p, uint32_t sums_s, uint32_t set_bytes, int rank,
                                               int tile, int nl, int lane, int part, int parts) {
  const int quads = (p.M + 3) / 4;
  const int first = quads * rank / p.cluster, last = quads * (rank + 1) / p.cluster;
  for (int q = first + part; q < last; q += parts) {
    float4 sum = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int r = 0; r < p.cluster; r += 2) {  // two CTAs' loads in flight
      float4 x[2][SETS];
#pragma unroll
      for (int u = 0; u < 2; ++u)
#pragma unroll
        for (int t = 0; t < SETS; ++t)
          if (r + u < p.cluster)
            x[u][t] = cluster_load4(sums_s + (uint32_t)t * set_bytes + (uint32_t)(q * 2048 + nl * 16), r + u);
#pragma unroll
      for (int u = 0; u < 2; ++u)
#pragma unroll
        for (int t = 0; t < SETS; ++t)
          if (r + u < p.cluster) {
            sum.x += x[u][t].x; sum.y += x[u][t].y; sum.z += x[u][t].z; sum.w += x[u][t].w;
          }
    }
    batch_store4<ACT>(p, tile * 128 + nl, lane, q * 4, sum);
  }
}

// Lane i's count says whether this warp's i-th 16-row chunk (chunk part + i * parts) of the tile's sums is
// complete; the complete ones are converted, written to C and put back to zero.
template <int ACT>
__device__ __forceinline__ void batch_finish(const BatchParams& p, int tile, int len, int wq, int lane, int part, int parts) {
  const int nl = wq * 32 + lane, n = tile * 128 + nl;
  float4* sums = reinterpret_cast<float4*>(p.partial) + (size_t)tile * (p.rows * 32) + nl;  // [rows / 4][128] quads
  int complete = 0;
  const int chunk = part + lane * parts;
  __syncwarp();
  if (chunk * 16 < p.M) {
    int* counter = p.chunk_counters + tile * 32 + wq * 8 + chunk;
    __threadfence();  // cumulative over the warp's additions (ordered by the barrier above)
    complete = atomicAdd(counter, len) + len == p.G ? 1 : 0;
    if (complete) {
      *counter = 0;
      __threadfence();
    }
  }
  unsigned mask = __ballot_sync(0xffffffffu, complete);
  while (mask) {
    const int mc0 = (part + (__ffs(mask) - 1) * parts) * 4;
    mask &= mask - 1;
    float4 x[4];  // independent loads
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if ((mc0 + u) * 4 < p.M) x[u] = __ldcg(sums + (mc0 + u) * 128);
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if ((mc0 + u) * 4 < p.M) {
        __stcg(sums + (mc0 + u) * 128, make_float4(0.f, 0.f, 0.f, 0.f));
        batch_store4<ACT>(p, n, lane, (mc0 + u) * 4, x[u]);
      }
  }
}

}  // namespace b200q
