// The two products of routed experts (see moe.cu) on the 5th-generation tensor cores, for bfloat16 and more than a
// few (token, expert) pairs a step.
//
// The weights are the 128-row operand of tcgen05.mma and the pairs the narrow one: a tile is 2 x 128 weight rows
// (gate and up rows of 128 features; or 256 rows of W_down) by up to 128 pairs of one expert, and the instruction's
// width is the tile's own number of pairs rounded up to 16, so an expert's ragged last tile costs no more than its
// pairs.  Accumulators of two tiles (2 x 2 x 128 columns) fill tensor memory: the epilogue of one runs under the
// products of the next.  A lane of the accumulator is a weight row, so a warp's stores of one pair are 32
// neighbouring features.
//   warp 0: TMA producer of the weights (and of W_down's input, whose rows lie in the pairs' order);
//   warp 1: tensor memory and tcgen05.mma;  warps 2-5: epilogue;
//   warps 6-9 (first product only): the pairs' tokens, gathered row by row with cp.async into the 128-byte swizzle
//   that the instruction reads.  (TMA's gather takes four rows a request, and a request costs the issuing warp
//   about 140 cycles: 32 of them a step of 64 against the step's 420 cycles of products.)
// Persistent: CTA b takes the tiles b, b + gridDim.x, ...; tiles of pairs first, so that the tiles of one expert
// that share a weight panel run side by side and the panel comes from HBM once.
//
// What bounds it: 2,048 tokens x top 4 of 32, 2048 -> 1024 -> 2048, is 103 GFLOP and 403 MB of weights, 62 us
// either way; the two kernels and the sort take 152 us (the mma.sync tiles of moe.cu: 485 us).  A step of 64 k of a whole tile
// writes 48 KB into shared memory and its products read 64 KB of it (the pairs for either panel), in 512 cycles of tensor
// work: some 220 bytes a cycle, where L2 brings 96.  200 tokens (800 pairs),
// where the weights are the bound: 83 us, 4.9 TB/s, against 141 us; 24 tokens: 76 against 125 us.  The sums' order over
// k is the tensor core's own in both forms; their results agreed bit for bit wherever they were compared.
// Every wait on an mbarrier is bounded (bit 16 of the error word), as in gemm_tcgen05.cu.
#include "tcgen05.cuh"
#include <math.h>

#define MT_PANEL (128 * 64 * 2)          // bytes of 128 rows x 64 of k
#define MT_STAGE (3 * MT_PANEL)          // two weight panels, one panel of pairs
#define MT_STAGES 4
#define MT_SMEM (MT_STAGES * MT_STAGE + 1024 + 256)

struct MoeTile { int e, r0, rows; };

// tile mt of the list: its rows end where the expert's next tile begins, or with the expert's pairs
__device__ __forceinline__ MoeTile moe_tile(const int* tile_expert, const int* tile_row0, const int* offsets, int mt,
                                            int m_tiles) {
  MoeTile t;
  t.e = tile_expert[mt];
  t.r0 = tile_row0[mt];
  const int end = (mt + 1 < m_tiles && tile_expert[mt + 1] == t.e) ? tile_row0[mt + 1] : offsets[t.e + 1];
  t.rows = min(end - t.r0, 128);
  return t;
}

__device__ __forceinline__ float moe_act(float g, float u, const GateAct& ga) {
  const float gg = fminf(g, ga.limit), uu = fminf(fmaxf(u, -ga.limit), ga.limit);
  return gg * (1.0f / (1.0f + expf(-ga.slope * gg))) * (uu + ga.shift);
}

// v[j]: this lane's feature of pair j.  Two pairs at a time: neighbouring lanes swap halves, so that a lane stores two
// features of one pair (4 bytes; 16 lanes are 64 contiguous bytes).  row(j) gives pair j's output row.
template <typename RowOf>
__device__ __forceinline__ void moe_store32(const float (&v)[32], bf16* out, int f, int n_out, int c0, int rows,
                                            int lane, RowOf row) {
  const int odd = lane & 1;
#pragma unroll
  for (int j = 0; j < 32; j += 2) {
    const float other = __shfl_xor_sync(0xffffffffu, odd ? v[j] : v[j + 1], 1);
    const __nv_bfloat162 p = odd ? __floats2bfloat162_rn(other, v[j + 1]) : __floats2bfloat162_rn(v[j], other);
    const size_t r = row(j + odd);
    if (c0 + j + odd < rows && (f & ~1) + 1 < n_out) *(__nv_bfloat162*)(out + r * n_out + (f & ~1)) = p;
  }
}

// GATE: out[r0 + j, f] = act of rows e 2F + f and e 2F + F + f of w with token sorted[r0 + j] / top of h.
// else: out[sorted[r0 + j], n] = row e N + n of w with row r0 + j of the map_b matrix.
template <bool GATE>
__global__ void __launch_bounds__(GATE ? 320 : 192)
moe_tcgen05_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_b, const bf16* h,
                   bf16* out, const int* offsets, const int* sorted, const int* tile_expert, const int* tile_row0,
                   const int* meta, int K, int n_out, int tiles_f, int top, GateAct ga, int* err) {
  constexpr int FT = GATE ? 128 : 256;                  // output features of a tile
  extern __shared__ unsigned char mt_raw[];
  unsigned char* base = (unsigned char*)(((uintptr_t)mt_raw + 1023) & ~(uintptr_t)1023);
  unsigned long long* bars = (unsigned long long*)(base + MT_STAGES * MT_STAGE);
  unsigned long long* full = bars;                      // [STAGES] operands -> MMA
  unsigned long long* empty = bars + MT_STAGES;         // [STAGES] MMA -> operands
  unsigned long long* acc_full = bars + 2 * MT_STAGES;  // [2]      MMA -> epilogue
  unsigned long long* acc_empty = acc_full + 2;         // [2]      epilogue -> MMA
  unsigned* tmem_slot = (unsigned*)(acc_empty + 2);
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const int num_kb = (K + 63) / 64;

  if (threadIdx.x == 0) {
    for (int i = 0; i < MT_STAGES; ++i) { mbar_init(&full[i], GATE ? 129 : 1); mbar_init(&empty[i], 1); }
    for (int i = 0; i < 2; ++i) { mbar_init(&acc_full[i], 1); mbar_init(&acc_empty[i], 4); }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"((unsigned long long)&map_w) : "memory");
    if (!GATE) asm volatile("prefetch.tensormap [%0];" ::"l"((unsigned long long)&map_b) : "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tg_smem(tmem_slot)), "r"(512) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const unsigned tmem_base = __shfl_sync(0xffffffffu, *tmem_slot, 0);
  pdl_wait_on(h, offsets, sorted, tile_expert, tile_row0, meta);
  pdl_launch();
  const int m_tiles = meta[0];
  const int num_tiles = __shfl_sync(0xffffffffu, m_tiles * tiles_f, 0);

  if (warp == 0) {
    if (lane == 0) {
      unsigned it = 0;
      bool ok = true;
      for (int tile = blockIdx.x; tile < num_tiles && ok; tile += gridDim.x) {
        const MoeTile t = moe_tile(tile_expert, tile_row0, offsets, tile % m_tiles, m_tiles);
        const int f0 = (tile / m_tiles) * FT;
        const int wa = t.e * (GATE ? 2 * n_out : n_out) + f0, wb = wa + (GATE ? n_out : 128);
        for (int kb = 0; kb < num_kb; ++kb, ++it) {
          const int s = it % MT_STAGES;
          ok = mbar_wait(&empty[s], ((it / MT_STAGES) & 1) ^ 1, err);   // a fresh barrier passes the wait for parity 1
          if (!ok) break;
          unsigned char* sa = base + s * MT_STAGE;
          mbar_expect_tx(&full[s], GATE ? 2 * MT_PANEL : 3 * MT_PANEL);
          tma_load_2d(sa, &map_w, kb * 64, wa, &full[s]);
          tma_load_2d(sa + MT_PANEL, &map_w, kb * 64, wb, &full[s]);
          if (!GATE) tma_load_2d(sa + 2 * MT_PANEL, &map_b, kb * 64, t.r0, &full[s]);
        }
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    // The whole warp walks and one lane issues, with what the instructions take from lane 0, and the next stage is looked at
    // ahead: see gemm_tcgen05.cu.
    int s = 0;
    unsigned phase = 0, ti = 0;
    bool ok = true, ready = false;
    for (int tile = blockIdx.x; tile < num_tiles && ok; tile += gridDim.x, ++ti) {
      const MoeTile t = moe_tile(tile_expert, tile_row0, offsets, tile % m_tiles, m_tiles);
      // instruction descriptor: float32 accumulate, bfloat16 A and B, both K-major, M = 128, N = the tile's pairs
      const unsigned wide = __shfl_sync(0xffffffffu, (unsigned)((t.rows + 15) >> 4), 0);
      const unsigned idesc = (1u << 4) | (1u << 7) | (1u << 10) | (wide << 18) | ((128u >> 4) << 24);
      const unsigned buf = ti & 1, use = ti >> 1;
      ok = __all_sync(0xffffffffu, mbar_wait(&acc_empty[buf], (use & 1) ^ 1, err));
      if (!ok) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const unsigned acc = tmem_base + buf * 256;
      for (int kb = 0; kb < num_kb; ++kb) {
        if (!ready) ok = __all_sync(0xffffffffu, mbar_wait(&full[s], phase, err));
        if (!ok) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        // The gathered rows were written by cp.async, and the instructions read them through the async proxy.  (Each stage
        // arrives with its copies; handed over by the copying warps when the second stage behind it was on its way, with the
        // fence there: 2,048 tokens, top 4 of 32, 162.7 us, so 159.6; top 2 of 16, 1,024 wide 84.3 -> 81.4.)
        if (GATE) asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        unsigned char* sa = base + s * MT_STAGE;
        const unsigned long long d0 = umma_desc(sa), d1 = umma_desc(sa + MT_PANEL), db = umma_desc(sa + 2 * MT_PANEL);
        unsigned long long* const here = &empty[s];
        if (++s == MT_STAGES) { s = 0; phase ^= 1; }
        ready = __all_sync(0xffffffffu, mbar_test(&full[s], phase));
        if (umma_elect()) {
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            umma_bf16(acc, d0 + 2 * k, db + 2 * k, idesc, (kb | k) != 0);
            umma_bf16(acc + 128, d1 + 2 * k, db + 2 * k, idesc, (kb | k) != 0);
          }
          umma_commit(here);
        }
        __syncwarp();
      }
      if (ok && umma_elect()) umma_commit(&acc_full[buf]);
      __syncwarp();
    }
  } else if (warp < 6) {
    const int quarter = warp & 3;
    unsigned ti = 0;
    bool ok = true;
    for (int tile = blockIdx.x; tile < num_tiles && ok; tile += gridDim.x, ++ti) {
      const MoeTile t = moe_tile(tile_expert, tile_row0, offsets, tile % m_tiles, m_tiles);
      const int f = (tile / m_tiles) * FT + quarter * 32 + lane;
      const unsigned buf = ti & 1, use = ti >> 1;
      ok = mbar_wait(&acc_full[buf], use & 1, err);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const unsigned addr = tmem_base + buf * 256 + ((unsigned)(quarter * 32) << 16);
#pragma unroll 1
      for (int c0 = 0; c0 < t.rows; c0 += 32) {
        unsigned a[32], b[32];
        tmem_ld32(addr + c0, a);
        tmem_ld32(addr + 128 + c0, b);
        const int mine = (c0 + lane < t.rows && !GATE) ? sorted[t.r0 + c0 + lane] : 0;
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
        float v[32];
        if (GATE) {
#pragma unroll
          for (int j = 0; j < 32; ++j) v[j] = moe_act(__uint_as_float(a[j]), __uint_as_float(b[j]), ga);
          moe_store32(v, out, f, n_out, c0, t.rows, lane, [&](int j) { return (size_t)(t.r0 + c0 + j); });
        } else {
          auto row = [&](int j) { return (size_t)__shfl_sync(0xffffffffu, mine, j); };
#pragma unroll
          for (int j = 0; j < 32; ++j) v[j] = __uint_as_float(a[j]);
          moe_store32(v, out, f, n_out, c0, t.rows, lane, row);
#pragma unroll
          for (int j = 0; j < 32; ++j) v[j] = __uint_as_float(b[j]);
          moe_store32(v, out, f + 128, n_out, c0, t.rows, lane, row);
        }
      }
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(&acc_empty[buf]);
    }
  } else if (GATE) {
    // thread: one 16-byte chunk of k of the rows g, g + 16, ... of the tile; eight neighbouring lanes a row's 128 bytes
    const int tid = threadIdx.x - 192, chunk = tid & 7, g = tid >> 3;
    unsigned it = 0;
    bool ok = true;
    for (int tile = blockIdx.x; tile < num_tiles && ok; tile += gridDim.x) {
      const MoeTile t = moe_tile(tile_expert, tile_row0, offsets, tile % m_tiles, m_tiles);
      const bf16* src[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const int r = g + 16 * i;
        src[i] = r < t.rows ? h + (size_t)(sorted[t.r0 + r] / top) * K + chunk * 8 : nullptr;
      }
      for (int kb = 0; kb < num_kb; ++kb, ++it) {
        const int s = it % MT_STAGES;
        ok = mbar_wait(&empty[s], ((it / MT_STAGES) & 1) ^ 1, err);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        const unsigned dst = tg_smem(base + s * MT_STAGE + 2 * MT_PANEL) + g * 128 + ((chunk ^ (g & 7)) << 4);
        const int n = kb * 64 + chunk * 8 < K ? 16 : 0;       // behind K: zeros
#pragma unroll
        for (int i = 0; i < 8; ++i)
          if (src[i])                                         // rows behind the tile's pairs: columns no one reads
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst + i * 2048), "l"(n ? src[i] + kb * 64 : src[i]), "r"(n) : "memory");
        // this thread's arrival, when its copies have landed
        asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(tg_smem(&full[s])) : "memory");
      }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 1)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512) : "memory");
}

template <bool GATE>
static int moe_tcgen05_launch(const CUtensorMap& mw, const CUtensorMap& mb, const void* h, void* out, const int* offsets,
                              const int* sorted, const int* tile_expert, const int* tile_row0, const int* meta,
                              int max_tiles, int K, int n_out, int top, GateAct ga, int* err, cudaStream_t stream) {
  static SmemLimit limit;
  if (const int e = limit.allow(moe_tcgen05_kernel<GATE>, MT_SMEM)) return e;
  const int tiles_f = (n_out + (GATE ? 127 : 255)) / (GATE ? 128 : 256);
  const long long tiles = (long long)max_tiles * tiles_f;
  if (tiles > (1ll << 30)) return RLLM_E_UNSUPPORTED;
  const int sms = tg_num_sms();
  rllm_launch_pdl(moe_tcgen05_kernel<GATE>, dim3((unsigned)(tiles < sms ? tiles : sms)), dim3(GATE ? 320 : 192),
                  (size_t)MT_SMEM, stream, mw, mb, (const bf16*)h, (bf16*)out, offsets, sorted, tile_expert, tile_row0,
                  meta, K, n_out, tiles_f, top, ga, err);
  RLLM_LAUNCH_CHECK();
  return 0;
}

// The experts' two products over the list that rllm_moe_sort made with tiles of 128 pairs.  y [pairs, F] holds the
// activations in the pairs' order.  H and F multiples of 8, 16-byte aligned pointers.
RLLM_EXPORT int rllm_moe_experts_tcgen05(const void* h, const void* w_gate_up, const void* w_down, void* y, void* out,
                                         const int* offsets, const int* sorted, const int* tile_expert,
                                         const int* tile_row0, const int* meta, int max_tiles, int pairs, int experts,
                                         int H, int F, int top, float limit, float alpha, float up_shift, int* err,
                                         cudaStream_t stream) {
  if (max_tiles <= 0 || pairs <= 0) return 0;
  if (H <= 0 || F <= 0 || top <= 0 || experts <= 0 || !err) return RLLM_E_BADARG;
  if (H % 8 || F % 8 || (((uintptr_t)h | (uintptr_t)w_gate_up | (uintptr_t)w_down | (uintptr_t)y | (uintptr_t)out) & 15))
    return RLLM_E_UNSUPPORTED;
  if ((long long)experts * 2 * F > (1ll << 30) || (long long)experts * H > (1ll << 30)) return RLLM_E_UNSUPPORTED;
  CUtensorMap mg, md, my;
  int rc = tg_make_map(&mg, w_gate_up, experts * 2 * F, H, H, 128);
  if (!rc) rc = tg_make_map(&md, w_down, experts * H, F, F, 128);
  if (!rc) rc = tg_make_map(&my, y, pairs, F, F, 128);
  if (rc) return rc;
  const GateAct ga{limit, alpha, up_shift};
  rc = moe_tcgen05_launch<true>(mg, mg, h, y, offsets, sorted, tile_expert, tile_row0, meta, max_tiles, H, F, top, ga,
                                err, stream);
  if (rc) return rc;
  return moe_tcgen05_launch<false>(md, my, nullptr, out, offsets, sorted, tile_expert, tile_row0, meta, max_tiles, F, H,
                                   top, ga, err, stream);
}
