// C[M, N] = A[M, K] . W[N, K]^T in bfloat16 on the 5th-generation tensor cores
// of sm_100a: the projections of prompt portions (M > 16 rows).
//
//   * operands come from global memory by TMA (cp.async.bulk.tensor, 128-byte
//     swizzle) into a ring of shared-memory stages, signalled by mbarriers;
//   * one elected thread issues tcgen05.mma (128 x BN x 16 per instruction,
//     operands described by shared-memory matrix descriptors), accumulating in
//     float32 in tensor memory (TMEM, BN columns of the 512);
//   * tcgen05.commit hands a stage back to the TMA producer when the MMAs that
//     read it are done, and at the end tells the epilogue warps that the
//     accumulator is complete;
//   * eight epilogue warps (two a quarter of the 128 lanes) read their 32 TMEM lanes with tcgen05.ld, round to
//     bfloat16 (or keep float32) and store; with the SiLU-gate epilogue the tile
//     holds 128 gate and 128 up features of [Wgate; Wup] side by side and
//     silu(gate) * up is applied to the accumulators
//     (crates/rllm-model/src/layers.rs:214-220), so the [T, 2I] intermediate
//     never exists.
// Warp 0: TMA producer.  Warp 1: TMEM allocation and MMA issue.  Warps 2-9:
// epilogue.  The kernel is persistent (one CTA per SM walks over output tiles) and
// keeps two accumulators in TMEM, so that the epilogue of a tile overlaps the
// MMAs of the next.  No multicast.  Larger products run on pairs of CTAs (cta_group::2) that share a tile of 256 rows:
// gemm_tcgen05_pair_kernel below.
//
// Every wait on an mbarrier is bounded: after the limit the thread sets bit 16
// of the error word and the CTA winds down (gives its TMEM columns back) instead
// of hanging.
//
// The reference computes these products with a library call
// (crates/rllm-model/src/layers.rs:162-175).
#include "tcgen05.cuh"
#include <math.h>

#define TG_BM 128
#define TG_BK 64
#define TG_EPI_WARPS 8                  // two a quarter of the lanes, half of the columns each
#define TG_THREADS (64 + 32 * TG_EPI_WARPS)
#define TG_EPI_BF16 0
#define TG_EPI_F32 1
#define TG_EPI_SILU 2
template <int BN> constexpr int tg_stages() { return BN == 256 ? 4 : (BN == 192 ? 5 : 6); }
// TMEM columns for two accumulators of BN columns: a power of two
template <int BN> constexpr int tg_tmem_cols() { return BN > 128 ? 512 : 256; }
template <int BN> constexpr int tg_stage_bytes() { return (TG_BM + BN) * TG_BK * 2; }
template <int BN> constexpr int tg_smem_bytes() { return tg_stages<BN>() * tg_stage_bytes<BN>() + 1024 + 256; }

// One warp's 32 rows and half of a tile's columns: from tensor memory (lane_addr: its lanes' first column) to row m,
// columns n0 .. of out.
template <int BN, int EPI>
__device__ __forceinline__ void tg_epilogue(unsigned lane_addr, int half, void* __restrict__ out, size_t at, int ldo, int m, int n0,
                                            int M, int N, const GateAct& ga) {
  constexpr int NOUT = (EPI == TG_EPI_SILU) ? BN / 2 : BN, SPLIT = NOUT / 64 * 32;      // 192 columns: 96 and 96
#pragma unroll 1
  for (int c0 = half ? SPLIT : 0; c0 < (half ? NOUT : SPLIT); c0 += 32) {
    unsigned r[32];
    tmem_ld32(lane_addr + c0, r);
    if (EPI == TG_EPI_SILU) {
      unsigned u[32];
      tmem_ld32(lane_addr + NOUT + c0, u);
      asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
      for (int j = 0; j < 32; ++j) {
        const float g = fminf(__uint_as_float(r[j]), ga.limit);
        const float up = fminf(fmaxf(__uint_as_float(u[j]), -ga.limit), ga.limit);
        r[j] = __float_as_uint(__fdividef(g, 1.0f + __expf(-ga.slope * g)) * (up + ga.shift));
      }
    } else {
      asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
    }
    if (m < M) {
      const int n = n0 + c0;
      if (EPI == TG_EPI_F32) {
        float* o = (float*)out + at + (size_t)m * ldo + n;
        if (n + 32 <= N && (((uintptr_t)o) & 15) == 0) {
#pragma unroll
          for (int j = 0; j < 32; j += 4)
            *(float4*)(o + j) = make_float4(__uint_as_float(r[j]), __uint_as_float(r[j + 1]),
                                            __uint_as_float(r[j + 2]), __uint_as_float(r[j + 3]));
        } else {
          for (int j = 0; j < 32; ++j) if (n + j < N) o[j] = __uint_as_float(r[j]);
        }
      } else {
        bf16* o = (bf16*)out + at + (size_t)m * ldo + n;
        if (n + 32 <= N && (((uintptr_t)o) & 15) == 0) {
#pragma unroll
          for (int j = 0; j < 32; j += 8) {
            uint4 v;
            __nv_bfloat162* p = (__nv_bfloat162*)&v;
#pragma unroll
            for (int q = 0; q < 4; ++q)
              p[q] = __floats2bfloat162_rn(__uint_as_float(r[j + 2 * q]), __uint_as_float(r[j + 2 * q + 1]));
            *(uint4*)(o + j) = v;
          }
        } else {
          for (int j = 0; j < 32; ++j) if (n + j < N) o[j] = __float2bfloat16_rn(__uint_as_float(r[j]));
        }
      }
    }
  }
}

// EPI: 0 bfloat16 out, 1 float32 out, 2 SiLU-gate (half of BN columns are gate rows; W rows n and up_offset + n pair up).
// Persistent: CTA b takes the output tiles b, b + gridDim.x, ... (rows of tiles first, so that CTAs
// running side by side share a weight tile in L2).  Two accumulators in TMEM: the epilogue of a
// tile runs while the tensor cores work on the next.
// HEADS: tiles_m x tiles_n tiles of every one of several products; A, W and out of product h lie h head strides further
// (the maps' third coordinate; c_head).
template <int BN, int EPI, bool HEADS>
__global__ void __launch_bounds__(TG_THREADS)
gemm_tcgen05_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_w,
                    void* __restrict__ out, int ldo, int M, int N, int K, int up_offset, int tiles_m,
                    int num_tiles, int* __restrict__ err, GateAct ga, int tiles_n, long long c_head) {
  constexpr int STAGES = tg_stages<BN>();
  constexpr int NOUT = (EPI == TG_EPI_SILU) ? BN / 2 : BN;     // output columns of a tile
  extern __shared__ unsigned char tg_raw[];
  unsigned char* base = (unsigned char*)(((uintptr_t)tg_raw + 1023) & ~(uintptr_t)1023);
  unsigned char* stage_mem = base;
  unsigned long long* bars = (unsigned long long*)(base + STAGES * tg_stage_bytes<BN>());
  unsigned long long* full = bars;                   // [STAGES]  TMA -> MMA
  unsigned long long* empty = bars + STAGES;         // [STAGES]  MMA -> TMA
  unsigned long long* acc_full = bars + 2 * STAGES;  // [2]       MMA -> epilogue
  unsigned long long* acc_empty = acc_full + 2;      // [2]       epilogue -> MMA
  unsigned* tmem_slot = (unsigned*)(acc_empty + 2);
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const int num_kb = (K + TG_BK - 1) / TG_BK;

  if (threadIdx.x == 0) {
    for (int i = 0; i < STAGES; ++i) { mbar_init(&full[i], 1); mbar_init(&empty[i], 1); }
    for (int i = 0; i < 2; ++i) { mbar_init(&acc_full[i], 1); mbar_init(&acc_empty[i], TG_EPI_WARPS); }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"((unsigned long long)&map_a) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"((unsigned long long)&map_w) : "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tg_smem(tmem_slot)), "r"(tg_tmem_cols<BN>()) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const unsigned tmem_base = __shfl_sync(0xffffffffu, *tmem_slot, 0);
  pdl_wait();                                        // what lies above overlaps the kernel ahead; nothing of global memory is read there
  pdl_launch();

  if (warp == 0) {
    if (lane == 0) {
      int s = -1;
      unsigned phase = 1;                                  // a fresh barrier passes the wait for parity 1
      bool ok = true;
      for (int tile = blockIdx.x; tile < num_tiles && ok; tile += gridDim.x) {
        const int m0 = (tile % tiles_m) * TG_BM, tn = tile / tiles_m, n0 = (HEADS ? tn % tiles_n : tn) * NOUT;
        const int head = HEADS ? tn / tiles_n : 0;
        for (int kb = 0; kb < num_kb; ++kb) {
          if (++s == STAGES) { s = 0; phase ^= 1; }
          ok = mbar_wait(&empty[s], phase, err);
          if (!ok) break;
          unsigned char* sa = stage_mem + s * tg_stage_bytes<BN>();
          unsigned char* sb = sa + TG_BM * TG_BK * 2;
          mbar_expect_tx(&full[s], (unsigned)tg_stage_bytes<BN>());
          if (HEADS) {
            tma_load_3d(sa, &map_a, kb * TG_BK, m0, head, &full[s]);
            tma_load_3d(sb, &map_w, kb * TG_BK, n0, head, &full[s]);
            continue;
          }
          tma_load_2d(sa, &map_a, kb * TG_BK, m0, &full[s]);
          if (EPI == TG_EPI_SILU) {
            tma_load_2d(sb, &map_w, kb * TG_BK, n0, &full[s]);
            tma_load_2d(sb + (BN / 2) * TG_BK * 2, &map_w, kb * TG_BK, up_offset + n0, &full[s]);
          } else {
            tma_load_2d(sb, &map_w, kb * TG_BK, n0, &full[s]);
          }
        }
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    // instruction descriptor: float32 accumulate, bfloat16 A and B, both K-major, N = BN, M = 128
    const unsigned idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((unsigned)(BN >> 3) << 17) | ((unsigned)(TG_BM >> 4) << 24);
    // The whole warp walks and one lane issues, with the warp's number and the accumulator's address taken from lane 0:
    // the compiler then knows the instruction's operands to be the same in all lanes, and a product costs the warp half
    // of the 100 cycles that a lane on its own took (tiles of 128 columns, 1,024 x 2,048 x 8,192: 40.5 -> 31.5 us, pairs
    // 39.1 -> 28.8; of 256 columns unchanged: a step there brings 48 KB into shared memory and reads them, 40 in a pair's
    // CTA, 135 to 140 bytes a cycle of both together, whichever of the two sets the pace).  The next stage's barrier is
    // looked at before this stage's products are issued, so that the answer is there afterwards.
    int s = 0;
    unsigned phase = 0, ti = 0;
    bool ok = true, ready = false;
    for (int tile = blockIdx.x; tile < num_tiles && ok; tile += gridDim.x, ++ti) {
      const unsigned buf = ti & 1, use = ti >> 1;
      ok = __all_sync(0xffffffffu, mbar_wait(&acc_empty[buf], (use & 1) ^ 1, err));   // the epilogue has drained this accumulator
      if (!ok) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const unsigned tmem_acc = tmem_base + buf * BN;
      for (int kb = 0; kb < num_kb; ++kb) {
        if (!ready) ok = __all_sync(0xffffffffu, mbar_wait(&full[s], phase, err));
        if (!ok) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        unsigned char* sa = stage_mem + s * tg_stage_bytes<BN>();
        unsigned char* sb = sa + TG_BM * TG_BK * 2;
        const unsigned long long da = umma_desc(sa), db = umma_desc(sb);
        unsigned long long* const here = &empty[s];
        if (++s == STAGES) { s = 0; phase ^= 1; }
        ready = __all_sync(0xffffffffu, mbar_test(&full[s], phase));
        if (umma_elect()) {
#pragma unroll
          for (int k = 0; k < TG_BK / 16; ++k)   // 16 bf16 = 32 bytes further along K: + 2 in the address field
            umma_bf16(tmem_acc, da + 2 * k, db + 2 * k, idesc, (kb | k) != 0);
          umma_commit(here);                     // the stage is free once these MMAs have read it
        }
        __syncwarp();
      }
      if (ok && umma_elect()) umma_commit(&acc_full[buf]);       // the accumulator is complete once all MMAs are done
      __syncwarp();
    }
    __syncwarp();
  } else {
    // epilogue: warp w reads TMEM lanes 32 (w % 4) .. + 31 = rows of the tile
    const int quarter = warp & 3;
    unsigned ti = 0;
    bool ok = true;
    for (int tile = blockIdx.x; tile < num_tiles && ok; tile += gridDim.x, ++ti) {
      const int m0 = (tile % tiles_m) * TG_BM, tn = tile / tiles_m, n0 = (HEADS ? tn % tiles_n : tn) * NOUT;
      const size_t at = HEADS ? (size_t)(tn / tiles_n) * c_head : 0;
      const unsigned buf = ti & 1, use = ti >> 1;
      const int m = m0 + quarter * 32 + lane;
      ok = mbar_wait(&acc_full[buf], use & 1, err);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const unsigned lane_addr = tmem_base + buf * BN + ((unsigned)(quarter * 32) << 16);
      tg_epilogue<BN, EPI>(lane_addr, (warp - 2) >> 2, out, at, ldo, m, n0, M, N, ga);
      // this warp has read its lanes of the accumulator: hand it back to the MMA warp
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(&acc_empty[buf]);
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 1) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(tg_tmem_cols<BN>()) : "memory");
  }
}

// ---------------------------------------------------------------------------
// The same product by pairs of CTAs (tcgen05 cta_group::2): a pair has a tile of 256 rows by BN columns, each CTA 128 of
// the rows.  The instruction takes its A operand from both CTAs (each its own rows) and its B operand half from each, so a
// CTA brings (128 + BN / 2) x 64 operand values a step of k instead of (128 + BN) x 64: a tile of 128 x 256 asks 96 bytes a
// cycle of L2 at the tensor cores' full rate, a pair's CTA 64.
//
// Both CTAs load their part (TMA, no multicast) into the same offsets of their own shared memory; the leader's (rank 0)
// barrier `full` counts the bytes of both.  The leader issues the instructions; tcgen05.commit arrives at both CTAs' `empty`
// and `acc_full`, and the epilogue warps of both arrive at the leader's `acc_empty`.  The pair leaves together: nothing
// arrives at a CTA that has gone.
// ---------------------------------------------------------------------------
#define TGP_BK 128                       // two panels of 64
template <int BN> constexpr int tgp_stage_bytes() { return (TG_BM + BN / 2) * TGP_BK * 2; }
template <int BN> constexpr int tgp_stages() { return BN == 128 ? 4 : 3; }
template <int BN> constexpr int tgp_smem_bytes() { return tgp_stages<BN>() * tgp_stage_bytes<BN>() + 1024 + 256; }

__device__ __forceinline__ unsigned tgp_rank() {
  unsigned r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
// the address of the leader's copy of a barrier
__device__ __forceinline__ unsigned tgp_leaders(const void* bar) {
  unsigned r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(r) : "r"(tg_smem(bar)));
  return r;
}
__device__ __forceinline__ void tgp_cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ void tgp_load_2d(void* dst, const CUtensorMap* map, int x, int y, unsigned leaders_bar) {
  asm volatile("cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
               ::"r"(tg_smem(dst)), "l"((unsigned long long)map), "r"(x), "r"(y), "r"(leaders_bar) : "memory");
}
__device__ __forceinline__ void tgp_umma(unsigned tmem_d, unsigned long long da, unsigned long long db, unsigned idesc, unsigned accumulate) {
  asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
               "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
               ::"r"(tmem_d), "l"(da), "l"(db), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void tgp_commit(void* bar) {      // at this barrier in both CTAs
  const unsigned short both = 3;
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
               ::"r"(tg_smem(bar)), "h"(both) : "memory");
}
// mbar_wait for barriers at which the other CTA's threads arrive
__device__ __forceinline__ bool tgp_wait(void* bar, unsigned parity, int* err) {
  const unsigned addr = tg_smem(bar);
  for (unsigned spin = 0; spin < TG_SPIN_LIMIT; ++spin) {
    unsigned done;
    asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
                 "selp.u32 %0, 1, 0, p;\n\t}" : "=r"(done) : "r"(addr), "r"(parity) : "memory");
    if (done) return true;
  }
  atomicOr(err, 16);
  return false;
}

template <int BN, int EPI>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(TG_THREADS)
gemm_tcgen05_pair_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_w,
                         void* __restrict__ out, int ldo, int M, int N, int K, int up_offset, int tiles_m, int num_tiles,
                         int* __restrict__ err, GateAct ga) {
  constexpr int STAGES = tgp_stages<BN>();
  constexpr int NOUT = (EPI == TG_EPI_SILU) ? BN / 2 : BN;     // output columns of a tile
  extern __shared__ unsigned char tg_raw[];
  unsigned char* base = (unsigned char*)(((uintptr_t)tg_raw + 1023) & ~(uintptr_t)1023);   // the same offset in both CTAs
  unsigned char* stage_mem = base;
  unsigned long long* bars = (unsigned long long*)(base + STAGES * tgp_stage_bytes<BN>());
  unsigned long long* full = bars;                   // [STAGES]  leader's: both CTAs' TMA -> MMA
  unsigned long long* empty = bars + STAGES;         // [STAGES]  MMA -> each CTA's TMA
  unsigned long long* acc_full = bars + 2 * STAGES;  // [2]       MMA -> each CTA's epilogue
  unsigned long long* acc_empty = acc_full + 2;      // [2]       leader's: both CTAs' epilogues -> MMA
  unsigned* tmem_slot = (unsigned*)(acc_empty + 2);
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const int rank = __shfl_sync(0xffffffffu, (int)tgp_rank(), 0), pair = blockIdx.x >> 1, pairs = gridDim.x >> 1;
  const int num_kb = (K + TGP_BK - 1) / TGP_BK;

  if (threadIdx.x == 0) {
    for (int i = 0; i < STAGES; ++i) { mbar_init(&full[i], 1); mbar_init(&empty[i], 1); }
    for (int i = 0; i < 2; ++i) { mbar_init(&acc_full[i], 1); mbar_init(&acc_empty[i], 2 * TG_EPI_WARPS); }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"((unsigned long long)&map_a) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"((unsigned long long)&map_w) : "memory");
  }
  __syncthreads();
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tg_smem(tmem_slot)), "r"(tg_tmem_cols<BN>()) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  tgp_cluster_sync();                                // both CTAs' barriers and tensor memory are there
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const unsigned tmem_base = __shfl_sync(0xffffffffu, *tmem_slot, 0);
  pdl_wait();                                        // what lies above overlaps the kernel ahead; nothing of global memory is read there
  pdl_launch();

  if (warp == 0) {
    if (lane == 0) {
      int s = -1;
      unsigned phase = 1, uses = 0;                      // a fresh barrier passes the wait for parity 1
      bool ok = true;
      for (int tile = pair; tile < num_tiles && ok; tile += pairs) {
        const int m0 = (tile % tiles_m) * 2 * TG_BM + rank * TG_BM, n0 = tile / tiles_m * NOUT;
        // this CTA's half of the weight rows: with the gate, rank 0 has the gate rows and rank 1 the up rows
        const int w0 = EPI == TG_EPI_SILU ? n0 + rank * up_offset : n0 + rank * (BN / 2);
        for (int kb = 0; kb < num_kb; ++kb, ++uses) {
          if (++s == STAGES) { s = 0; phase ^= 1; }
          ok = mbar_wait(&empty[s], phase, err);
          if (!ok) break;
          unsigned char* sa = stage_mem + s * tgp_stage_bytes<BN>();
          unsigned char* sb = sa + TG_BM * TGP_BK * 2;
          const int x = kb * TGP_BK;
          const bool two = x + 64 < K;                     // the second panel has values
          if (rank == 0) mbar_expect_tx(&full[s], (two ? 2u : 1u) * tgp_stage_bytes<BN>());
          const unsigned bar = tgp_leaders(&full[s]);
          tgp_load_2d(sa, &map_a, x, m0, bar);
          tgp_load_2d(sb, &map_w, x, w0, bar);
          if (two) {
            tgp_load_2d(sa + TG_BM * 128, &map_a, x + 64, m0, bar);
            tgp_load_2d(sb + BN / 2 * 128, &map_w, x + 64, w0, bar);
          }
        }
      }
      // the last uses of the stages: their commits have arrived here before this CTA leaves
      for (unsigned i = 1; i <= (unsigned)STAGES && i <= uses && ok; ++i)
        ok = mbar_wait(&empty[(uses - i) % STAGES], ((uses - i) / STAGES) & 1, err);
    }
    __syncwarp();
  } else if (warp == 1) {
    if (rank == 0) {
      // instruction descriptor: float32 accumulate, bfloat16 A and B, both K-major, N = BN, M = 256
      const unsigned idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((unsigned)(BN >> 3) << 17) | ((unsigned)(2 * TG_BM >> 4) << 24);
      int s = 0;
      unsigned phase = 0, ti = 0;
      bool ok = true, ready = false;
      for (int tile = pair; tile < num_tiles && ok; tile += pairs, ++ti) {
        const unsigned buf = ti & 1, use = ti >> 1;
        ok = __all_sync(0xffffffffu, tgp_wait(&acc_empty[buf], (use & 1) ^ 1, err));   // both epilogues have drained this accumulator
        if (!ok) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const unsigned tmem_acc = tmem_base + buf * BN;
        for (int kb = 0; kb < num_kb; ++kb) {
          if (!ready) ok = __all_sync(0xffffffffu, mbar_wait(&full[s], phase, err));
          if (!ok) break;
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          unsigned char* sa = stage_mem + s * tgp_stage_bytes<BN>();
          const unsigned long long da = umma_desc(sa), db = umma_desc(sa + TG_BM * TGP_BK * 2);
          unsigned long long* const here = &empty[s];
          if (++s == STAGES) { s = 0; phase ^= 1; }
          ready = __all_sync(0xffffffffu, mbar_test(&full[s], phase));      // the next stage's: see gemm_tcgen05_kernel
          if (umma_elect()) {
#pragma unroll
            for (int k = 0; k < 4; ++k)            // 16 bf16 = 32 bytes further along K: + 2 in the address field
              tgp_umma(tmem_acc, da + 2 * k, db + 2 * k, idesc, (kb | k) != 0);
            if (kb * TGP_BK + 64 < K) {
#pragma unroll
              for (int k = 0; k < 4; ++k)
                tgp_umma(tmem_acc, da + (TG_BM * 128 >> 4) + 2 * k, db + (BN / 2 * 128 >> 4) + 2 * k, idesc, 1u);
            }
            tgp_commit(here);
          }
          __syncwarp();
        }
        if (ok && umma_elect()) tgp_commit(&acc_full[buf]);
        __syncwarp();
      }
    }
    __syncwarp();
  } else {
    const int quarter = warp & 3;
    unsigned ti = 0;
    bool ok = true;
    for (int tile = pair; tile < num_tiles && ok; tile += pairs, ++ti) {
      const int m0 = (tile % tiles_m) * 2 * TG_BM + rank * TG_BM, n0 = tile / tiles_m * NOUT;
      const unsigned buf = ti & 1, use = ti >> 1;
      ok = __all_sync(0xffffffffu, mbar_wait(&acc_full[buf], use & 1, err));
      if (!ok) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      tg_epilogue<BN, EPI>(tmem_base + buf * BN + ((unsigned)(quarter * 32) << 16), (warp - 2) >> 2, out, (size_t)0, ldo, m0 + quarter * 32 + lane, n0, M, N, ga);
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0)
        asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(tgp_leaders(&acc_empty[buf])) : "memory");
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  tgp_cluster_sync();
  if (warp == 1) {
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(tg_tmem_cols<BN>()) : "memory");
  }
}

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------
// maps' boxes: TG_BM rows of A, NOUT rows of W
template <int BN, int EPI, bool HEADS>
static int tg_run(const CUtensorMap& ma, const CUtensorMap& mw, void* out, int ldo, int M, int N, int K, int up_offset,
                  int heads, long long c_head, int* err, cudaStream_t stream, GateAct ga) {
  constexpr int NOUT = (EPI == TG_EPI_SILU) ? BN / 2 : BN;
  static SmemLimit limit;
  if (const int e = limit.allow(gemm_tcgen05_kernel<BN, EPI, HEADS>, tg_smem_bytes<BN>())) return e;
  const int tiles_m = (M + TG_BM - 1) / TG_BM, tiles_n = (N + NOUT - 1) / NOUT;
  const long long num_tiles = (long long)tiles_m * tiles_n * heads;
  if (num_tiles > (1ll << 30)) return RLLM_E_UNSUPPORTED;
  const int num_sms = tg_num_sms();
  const int grid = (int)(num_tiles < num_sms ? num_tiles : num_sms);
  rllm_launch_pdl(gemm_tcgen05_kernel<BN, EPI, HEADS>, dim3(grid), dim3(TG_THREADS), (size_t)tg_smem_bytes<BN>(), stream, ma, mw, out,
                  ldo, M, N, K, up_offset, tiles_m, (int)num_tiles, err, ga, tiles_n, c_head);
  RLLM_LAUNCH_CHECK();
  return 0;
}

template <int BN, int EPI>
static int tgp_launch(const void* a, int lda, const void* w, int ldw, int w_rows, void* out, int ldo, int M, int N, int K,
                      int up_offset, int* err, cudaStream_t stream, GateAct ga) {
  constexpr int NOUT = (EPI == TG_EPI_SILU) ? BN / 2 : BN;
  CUtensorMap ma, mw;
  int rc = tg_make_map(&ma, a, M, K, lda, TG_BM);
  if (!rc) rc = tg_make_map(&mw, w, w_rows, K, ldw, BN / 2);
  if (rc) return rc;
  static SmemLimit limit;
  if (const int e = limit.allow(gemm_tcgen05_pair_kernel<BN, EPI>, tgp_smem_bytes<BN>())) return e;
  const int tiles_m = (M + 2 * TG_BM - 1) / (2 * TG_BM), tiles_n = (N + NOUT - 1) / NOUT;
  const long long num_tiles = (long long)tiles_m * tiles_n;
  if (num_tiles > (1ll << 29)) return RLLM_E_UNSUPPORTED;
  const int pairs = tg_num_sms() / 2;
  const int grid = 2 * (int)(num_tiles < pairs ? num_tiles : pairs);
  rllm_launch_pdl(gemm_tcgen05_pair_kernel<BN, EPI>, dim3(grid), dim3(TG_THREADS), (size_t)tgp_smem_bytes<BN>(), stream, ma, mw, out,
                  ldo, M, N, K, up_offset, tiles_m, (int)num_tiles, err, ga);
  RLLM_LAUNCH_CHECK();
  return 0;
}

template <int BN, int EPI>
static int tg_launch(const void* a, int lda, const void* w, int ldw, int w_rows, void* out, int ldo, int M, int N,
                     int K, int up_offset, int* err, cudaStream_t stream, GateAct ga) {
  constexpr int NOUT = (EPI == TG_EPI_SILU) ? BN / 2 : BN;
  CUtensorMap ma, mw;
  int rc = tg_make_map(&ma, a, M, K, lda, TG_BM);
  if (rc) return rc;
  rc = tg_make_map(&mw, w, w_rows, K, ldw, NOUT);
  if (rc) return rc;
  return tg_run<BN, EPI, false>(ma, mw, out, ldo, M, N, K, up_offset, 1, 0, err, stream, ga);
}

// Which form a product of `rows` rows takes, and how wide its tile is: the least estimated time, a launch + a step of 64 k
// times the steps times the rounds of the persistent CTAs, in microseconds (one launch after another on a B200):
//   CTAs on their own   4.6 + 0.37, 0.30 or 0.22 a step of 256, 192 or 128 columns
//   pairs               6.3 + 0.32, 6.0 + 0.275 or 5.8 + 0.19 (a tile of twice the rows; two cluster barriers more a launch)
// A step costs by the bytes that pass through shared memory, so narrow tiles pay where wide ones would leave the last round
// empty.  Measured, single 256 / 192 / 128 and pairs 256 / 192 / 128, M x N x K:
//   2,048 x 2,048 x 2,048 16.3 / 22.2 / 18.6, 16.7 / 21.3 / 17.2;    x 4,096 28.2 / 37.6 / 32.1, 26.6 / 37.6 / 28.7
//   2,047 x 3,072 x 2,048 30.5 / 24.4 / 27.4, 27.9 / 23.7 / 24.4;    700 x 3,072 x 2,048 17.6 / 14.1 / 11.6, 17.3 / 14.7 / 11.8
//   2,048 x 1,344 x 2,048 17.2 / 13.7 / 17.8, 17.2 / 14.0 / 16.2;    1,024 x 2,048 x 8,192 49 / 40 / 31.5, 42 / 39 / 28.8
//   6,327 x 3,072 x 2,048 69 / 67 / 76, 61 / 63 / 68
// (Products of fewer than ops.TCGEN05_MIN_TILES tiles of 128 x 256, as 700 x 3,072 x 2,048 and 1,024 x 2,048 x 8,192, come only
// from callers that ask for this kernel themselves: linear gives them to the library.)
// With the gate a tile has half as many output columns.
// Every column of tiles passes over A once more, from HBM where A is larger than what L2 (126 MB) keeps of it: tiles of 128
// are left out there unless one or two of them span all columns.  Pairs of 256 / 128 columns, M x N x K (A in MB): 8,192 x 1,344 x
// 8,192 (128) 142 / 161, 16,384 x 1,344 x 4,096 (128) 162 / 222, 16,384 x 1,344 x 8,192 (256) 312 / 426, 8,192 x 1,344 x 6,144 (96)
// 110 / 123, x 5,120 (80) 93 / 100, x 4,096 (64) 75 / 75; but 8,192 x 200 x 8,192 45 / 37.
struct TgForm { int width; bool pair; };
static TgForm tg_form(long long tiles_rows, long long tiles_rows2, int N, int K, bool gate, bool pairs, long long sms, long long a_bytes) {
  static const int widths[3] = {256, 192, 128};
  static const double single[2][3] = {{4.6, 4.6, 4.6}, {0.37, 0.30, 0.22}}, both[2][3] = {{6.3, 6.0, 5.8}, {0.32, 0.275, 0.19}};
  const double steps = (K + TG_BK - 1) / TG_BK;
  TgForm best{256, false};
  double least = 1e30;
  auto passes = [&](int i, long long across) { return widths[i] == 128 && across > 2 && a_bytes > 72ll << 20; };   // over A, too many
  for (int i = 0; i < 3; ++i) {
    const long long cols = gate ? widths[i] / 2 : widths[i], across = (N + cols - 1) / cols;
    if (passes(i, across)) continue;
    const double t = single[0][i] + single[1][i] * steps * (double)((tiles_rows * across + sms - 1) / sms);
    if (t < least) { least = t; best = TgForm{widths[i], false}; }
  }
  for (int i = 0; i < 3 && pairs && sms >= 2; ++i) {
    const long long cols = gate ? widths[i] / 2 : widths[i], across = (N + cols - 1) / cols;
    if (passes(i, across)) continue;
    const double t = both[0][i] + both[1][i] * steps * (double)((tiles_rows2 * across + sms / 2 - 1) / (sms / 2));
    if (t < least) { least = t; best = TgForm{widths[i], true}; }
  }
  return best;
}
static TgForm tg_form_of(int M, int N, int K, int epilogue, long long sms) {
  return tg_form((M + TG_BM - 1) / TG_BM, (M + 2 * TG_BM - 1) / (2 * TG_BM), N, K, epilogue == TG_EPI_SILU, true, sms,
                 2ll * M * K);
}
// the width of the tiles, negative for pairs (the host's rule alone, for tests)
RLLM_EXPORT int rllm_gemm_tcgen05_form(int M, int N, int K, int epilogue, int sms) {
  const TgForm f = tg_form_of(M, N, K, epilogue, sms);
  return f.pair ? -f.width : f.width;
}

// epilogue 0: out bfloat16 [M, N]; 1: out float32 [M, N]; 2: W = [gate rows (N); up rows (N)] stacked,
// out bfloat16 [M, N] = silu(A . gate^T) * (A . up^T), with the gate's constants limit, slope, shift (GateAct).  err:
// the engine's error word (bit 16: a wait ran out).
RLLM_EXPORT int rllm_gemm_tcgen05(const void* a, int lda, const void* w, int ldw, void* out, int ldo, int M, int N,
                                  int K, int epilogue, float limit, float slope, float shift, int* err,
                                  cudaStream_t stream) {
  if (M <= 0 || N <= 0) return 0;
  if (K <= 0 || lda < K || ldw < K || ldo < N || !err) return RLLM_E_BADARG;
  // TMA: 16-byte aligned bases and row strides
  if (K % 8 || lda % 8 || ldw % 8 || (((uintptr_t)a | (uintptr_t)w) & 15)) return RLLM_E_UNSUPPORTED;
  const TgForm form = tg_form_of(M, N, K, epilogue, tg_num_sms());
  const bool gate = epilogue == TG_EPI_SILU;
  const int w_rows = gate ? 2 * N : N, up = gate ? N : 0;
  const GateAct ga{limit, slope, shift};
#define TG_GO(F_, BN_, EPI_) return F_<BN_, EPI_>(a, lda, w, ldw, w_rows, out, ldo, M, N, K, up, err, stream, ga)
#define TG_BY_FORM(EPI_)                                                          \
  if (form.pair && form.width == 256) TG_GO(tgp_launch, 256, EPI_);              \
  if (form.pair && form.width == 192) TG_GO(tgp_launch, 192, EPI_);              \
  if (form.pair) TG_GO(tgp_launch, 128, EPI_);                                   \
  if (form.width == 256) TG_GO(tg_launch, 256, EPI_);                            \
  if (form.width == 192) TG_GO(tg_launch, 192, EPI_);                            \
  TG_GO(tg_launch, 128, EPI_)
  switch (epilogue) {
    case TG_EPI_BF16: TG_BY_FORM(TG_EPI_BF16);
    case TG_EPI_F32: TG_BY_FORM(TG_EPI_F32);
    case TG_EPI_SILU: TG_BY_FORM(TG_EPI_SILU);
  }
  return RLLM_E_BADARG;
}

template <int BN>
static int tg_launch_heads(const void* a, long long lda, long long a_head, const void* w, long long ldw, long long w_head,
                           void* out, int ldo, long long c_head, int M, int N, int K, int heads, int* err, cudaStream_t stream) {
  CUtensorMap ma, mw;
  int rc = tg_make_map3(&ma, a, M, K, lda, heads, a_head, TG_BM);
  if (!rc) rc = tg_make_map3(&mw, w, N, K, ldw, heads, w_head, BN);
  if (rc) return rc;
  return tg_run<BN, TG_EPI_BF16, true>(ma, mw, out, ldo, M, N, K, 0, heads, c_head, err, stream, GateAct{INFINITY, 1.f, 0.f});
}

// Several products at once, bfloat16: out[h] [M, N] = A[h] [M, K] . W[h] [N, K]^T, all strides in elements.
RLLM_EXPORT int rllm_head_gemm_tcgen05(const void* a, long long lda, long long a_head, const void* w, long long ldw,
                                       long long w_head, void* out, int ldo, long long c_head, int M, int N, int K, int heads,
                                       int* err, cudaStream_t stream) {
  if (M <= 0 || N <= 0 || heads <= 0) return 0;
  if (K <= 0 || !err) return RLLM_E_BADARG;
  if (K % 8 || lda % 8 || a_head % 8 || ldw % 8 || w_head % 8 || (((uintptr_t)a | (uintptr_t)w) & 15)) return RLLM_E_UNSUPPORTED;
  const int bn = tg_form((long long)((M + TG_BM - 1) / TG_BM) * heads, 0, N, K, false, false, tg_num_sms(), 2ll * M * K).width;
  if (bn == 256) return tg_launch_heads<256>(a, lda, a_head, w, ldw, w_head, out, ldo, c_head, M, N, K, heads, err, stream);
  if (bn == 192) return tg_launch_heads<192>(a, lda, a_head, w, ldw, w_head, out, ldo, c_head, M, N, K, heads, err, stream);
  return tg_launch_heads<128>(a, lda, a_head, w, ldw, w_head, out, ldo, c_head, M, N, K, heads, err, stream);
}
