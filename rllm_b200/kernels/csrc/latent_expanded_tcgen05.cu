// Latent attention of prompt portions with every head's own keys and values, bfloat16 on the tcgen05 tensor cores.
//
// A head's key is [W_uk[h] c | shared rotated part] and its value W_uv[h] c.  latent_attention_tcgen05.cu moves W_uk and
// W_uv to the query side and walks the cached rows: dk + dv = 1,088 multiplications a (query, key, head) at rows of 576.
// Here the visible rows are gathered from their pages (latent_attention.cu), one product makes all heads' keys and values
// of them, and a (query, key, head) costs nope + rot + v = 320 multiplications.  The product is paid once a visible row
// (2 kv_rank (nope + v) a head, as the query side's two products are a query): worth it while the rows are not many
// times the queries (the rule is latent_expanded_pays in ops.py).
//
// One CTA per (tile of 128 query tokens, head, sequence), two CTAs an SM; key tiles of BN at absolute positions.
//   warp 0     TMA: Q once, then a tile's K (panels of 64 dims: the head's own from `kv`, the shared one from the
//              gathered rows) and V panels; the rows lie one after the other, so a tile is NQ + DV / 64 requests.
//   warp 1     tensor memory (S: BN columns, output: DV, P: BN / 2) and the products: S = Q K^T, then output += P V with P
//              in tensor memory and V as the MN-major operand.
//   warps 2-9  softmax, two threads a row, as in attention_tcgen05.cu; the reference point is the running maximum, as in
//              latent_attention_tcgen05.cu.
// Measured, 2,048 tokens, 16 heads of 128 + 64 | 128 over rows of 512 + 64: attention 221 -> 39 us (550 TFLOP/s of visible
// pairs), gather 7 and product 16 us in place of the query side's products 21 + 16; the mixer 320 -> 120 us, its distance
// from float64 0.0052 -> 0.0051 of the result's norm.  The longest CTAs (32 tiles of keys, 1 us each) are what is left.
// K has two stages; V one or two, what the 113 KB of half an SM leave: V of a tile is asked for when the product of the
// tile before is through, which the tile's softmax hides.
// Every wait on an mbarrier is bounded (bit 16 of the error word, then wind-down).  No cluster, no multicast.
#include "attention_tcgen05.cuh"

#define LE_BM 128
#define LE_THREADS 320
#define LE_ALIGN 128             // a sequence's gathered rows begin at a multiple of it

template <int NQ, int DV> struct LeShape {
  static constexpr int BN = (NQ == 2 && DV == 64) ? 128 : 64;      // keys a tile
  static constexpr int PANEL = BN * 128;                           // bytes of 64 dims of a tile's keys
  static constexpr int K_STAGE = NQ * PANEL, V_STAGE = (DV / 64) * PANEL;
  static constexpr int FIXED = NQ * 16384 + 2 * K_STAGE;
  static constexpr int NV = FIXED + 2 * V_STAGE <= 114688 ? 2 : 1;
  static constexpr int SMEM = FIXED + NV * V_STAGE + 512;
};

// the oldest key that a query at position p sees
__device__ __forceinline__ int le_oldest(int p, int window) { return (window > 0 && p - window + 1 > 0) ? p - window + 1 : 0; }

template <int NQ, int DV>
__global__ void __launch_bounds__(LE_THREADS, 2)
latent_expanded_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_kv,
                       const __grid_constant__ CUtensorMap map_r, bf16* __restrict__ out, const int* __restrict__ q_start,
                       const int* __restrict__ seq_lens, int seq_begin, int seq_end, int heads, int rot, int window,
                       float scale_log2, const float* __restrict__ sink, int* __restrict__ err) {
  pdl_wait();
  using Shape = LeShape<NQ, DV>;
  constexpr int BN = Shape::BN, PANEL = Shape::PANEL, NV = Shape::NV, VP = DV / 64, NOPE = (NQ - 1) * 64;
  extern __shared__ __align__(1024) unsigned char le_raw[];
  unsigned char* base = le_raw;
  if (tg_smem(base) & 1023u) {                    // the swizzled tiles need 1024-byte alignment
    if (threadIdx.x == 0) atomicOr(err, 32);
    return;
  }
  unsigned char* sQ = base;                       // NQ panels x [128 rows][64 dims]
  unsigned char* sK = sQ + NQ * 16384;            // 2 stages x NQ panels x [BN keys][64 dims]
  unsigned char* sV = sK + 2 * Shape::K_STAGE;    // NV stages x VP panels x [BN keys][64 dims]
  unsigned long long* bars = (unsigned long long*)(sV + NV * Shape::V_STAGE);
  unsigned long long* q_full = bars;              // TMA -> MMA
  unsigned long long* k_full = bars + 1;          // [2] TMA -> MMA
  unsigned long long* k_empty = bars + 3;         // [2] MMA -> TMA
  unsigned long long* v_full = bars + 5;          // [2] TMA -> MMA (and the softmax warps)
  unsigned long long* v_empty = bars + 7;         // [2] MMA -> TMA
  unsigned long long* s_full = bars + 9;          // MMA -> softmax
  unsigned long long* p_full = bars + 10;         // softmax (8 warps) -> MMA
  unsigned long long* pv_full = bars + 11;        // MMA -> softmax
  unsigned long long* s_free = bars + 12;         // softmax (8 warps) -> MMA
  unsigned long long* xbar = bars + 13;           // [4] the two warps of a row quarter, one another
  unsigned* tmem_slot = (unsigned*)(bars + 17);
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const int head = blockIdx.x % heads;
  // which (sequence, tile): the tiles that see the most keys first; where the sequence's gathered rows begin
  int s = -1, tile = 0, row0 = 0;
  {
    int left = blockIdx.x / heads;
    for (int i = seq_begin; i < seq_end; ++i) {
      const int qn = q_start[i + 1] - q_start[i], n = (qn + LE_BM - 1) / LE_BM;
      if (left < n) { s = i; tile = n - 1 - left; break; }
      left -= n;
      row0 += seq_lens[i] - le_oldest(seq_lens[i] - qn, window) / LE_ALIGN * LE_ALIGN;
    }
  }
  if (s < 0) return;
  const int qs = q_start[s], qlen = q_start[s + 1] - qs;
  const int pos0 = seq_lens[s] - qlen;
  row0 -= le_oldest(pos0, window) / LE_ALIGN * LE_ALIGN;            // row of the sequence's key j: row0 + j
  const int t0 = tile * LE_BM;
  const int ntok = min(LE_BM, qlen - t0);
  const int first_pos = pos0 + t0, last_pos = pos0 + t0 + ntok - 1;
  const int kmin = le_oldest(first_pos, window), kend = last_pos + 1;
  const int tile_lo = kmin / BN, ntiles = (kend + BN - 1) / BN - tile_lo;

  if (threadIdx.x == 0) {
    mbar_init(q_full, 1);
    for (int i = 0; i < 2; ++i) { mbar_init(&k_full[i], 1); mbar_init(&k_empty[i], 1); mbar_init(&v_full[i], 1); mbar_init(&v_empty[i], 1); }
    mbar_init(s_full, 1);
    mbar_init(p_full, 8);
    mbar_init(pv_full, 1);
    mbar_init(s_free, 8);
    for (int i = 0; i < 4; ++i) mbar_init(&xbar[i], 2);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"((unsigned long long)&map_q) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"((unsigned long long)&map_kv) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"((unsigned long long)&map_r) : "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tg_smem(tmem_slot)), "r"(256) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  pdl_launch();                                   // behind the allocation: see pdl_launch
  const unsigned tmem_s = __shfl_sync(0xffffffffu, *tmem_slot, 0), tmem_o = tmem_s + BN, tmem_p = tmem_o + DV;   // BN + DV + BN / 2 <= 256 columns

  if (warp == 0) {
    if (lane == 0) {
      mbar_expect_tx(q_full, (unsigned)(NQ * 16384));
      for (int p = 0; p < NQ; ++p) tma_load_3d(sQ + p * 16384, &map_q, p * 64, head, qs + t0, q_full);
      const int kx = head * NOPE, vx = heads * NOPE + head * DV;
      int nk = 0, nv = 0;                          // tiles whose K, V have been asked for
      unsigned spin = 0;
      while (nk < ntiles || nv < ntiles) {
        bool some = false;
        if (nk < ntiles && mbar_test(&k_empty[nk & 1], ((nk >> 1) & 1) ^ 1)) {
          unsigned char* to = sK + (nk & 1) * Shape::K_STAGE;
          const int y = row0 + (tile_lo + nk) * BN;
          mbar_expect_tx(&k_full[nk & 1], (unsigned)Shape::K_STAGE);
          for (int p = 0; p < NQ - 1; ++p) tma_load_2d(to + p * PANEL, &map_kv, kx + p * 64, y, &k_full[nk & 1]);
          tma_load_2d(to + (NQ - 1) * PANEL, &map_r, 0, y, &k_full[nk & 1]);
          ++nk;
          some = true;
        }
        if (nv < nk && mbar_test(&v_empty[nv % NV], ((nv / NV) & 1) ^ 1)) {
          unsigned char* to = sV + (nv % NV) * Shape::V_STAGE;
          const int y = row0 + (tile_lo + nv) * BN;
          mbar_expect_tx(&v_full[nv % NV], (unsigned)Shape::V_STAGE);
          for (int p = 0; p < VP; ++p) tma_load_2d(to + p * PANEL, &map_kv, vx + p * 64, y, &v_full[nv % NV]);
          ++nv;
          some = true;
        }
        if (some) spin = 0;
        else if (++spin > TG_SPIN_LIMIT) { atomicOr(err, 16); break; }
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    // The whole warp walks and one lane issues, with what the instructions take from lane 0: the compiler then knows their
    // operands to be the same in all lanes, and a product costs the warp half as much (see gemm_tcgen05.cu; 45 -> 39 us).
    const unsigned idesc_s = (1u << 4) | (1u << 7) | (1u << 10) | ((unsigned)(BN >> 3) << 17) | ((unsigned)(LE_BM >> 4) << 24);
    const unsigned idesc_pv = (1u << 4) | (1u << 7) | (1u << 10) | (1u << 16) | ((unsigned)(DV >> 3) << 17) | ((unsigned)(LE_BM >> 4) << 24);
    const unsigned long long dq = umma_desc(sQ);
    const int rot_steps = (rot + 15) / 16;         // the shared part's dims behind `rot` are zeros
    const int tiles = __shfl_sync(0xffffffffu, ntiles, 0);
    auto scores = [&](int st) {
      const unsigned long long dk = umma_desc(sK + st * Shape::K_STAGE);
      if (umma_elect()) {
#pragma unroll
        for (int k = 0; k < NQ * 4; ++k) {
          if (k >= (NQ - 1) * 4 + rot_steps) break;
          umma_bf16(tmem_s, dq + (unsigned long long)((k >> 2) * (16384 >> 4) + 2 * (k & 3)),
                    dk + (unsigned long long)((k >> 2) * (PANEL >> 4) + 2 * (k & 3)), idesc_s, k != 0);
        }
        umma_commit(s_full);
        umma_commit(&k_empty[st]);
      }
      __syncwarp();
    };
    auto wait = [&](unsigned long long* bar, unsigned parity) { return __all_sync(0xffffffffu, mbar_wait(bar, parity, err)) != 0; };
    bool ok = wait(q_full, 0) && wait(&k_full[0], 0);
    if (ok) {
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      scores(0);
    }
    for (int it = 0; it < tiles && ok; ++it) {
      if (it + 1 < tiles) {                        // the next tile's scores, as soon as the softmax warps hold this tile's
        const int sn = (it + 1) & 1;
        ok = wait(&k_full[sn], ((it + 1) >> 1) & 1) && wait(s_free, it & 1);
        if (!ok) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        scores(sn);
      }
      const int sv = it % NV;
      ok = wait(&v_full[sv], (it / NV) & 1) && wait(p_full, it & 1);   // P is in tensor memory, O is rescaled
      if (!ok) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      // V: 64 dims x 8 keys a swizzle atom, 8 keys on 1024 bytes further (stride field), 64 dims on a panel further
      // (leading-dimension field)
      const unsigned long long dv = (umma_desc(sV + sv * Shape::V_STAGE) & ~(0x3FFFull << 16)) | ((unsigned long long)(PANEL >> 4) << 16);
      if (umma_elect()) {
#pragma unroll
        for (int kk = 0; kk < BN / 16; ++kk)
          umma_bf16_tmem_a(tmem_o, tmem_p + kk * 8, dv + (unsigned long long)(kk * (2048 >> 4)), idesc_pv, (it | kk) != 0);
        umma_commit(&v_empty[sv]);
        umma_commit(pv_full);
      }
      __syncwarp();
    }
  } else {
    const int quarter = warp & 3, half = (warp - 2) >> 2;
    const int r = quarter * 32 + lane;               // this thread's row of the tile
    // rows behind the portion's last token compute like the others; their result is not stored
    const int pos = first_pos + r;
    const int row_hi = pos + 1, row_lo = le_oldest(pos, window);
    const int clear_lo = le_oldest(first_pos + LE_BM - 1, window), clear_hi = first_pos + 1;   // tiles inside need no mask
    float m_ref = -INFINITY, l = 0.f;
    const unsigned lane_sel = (unsigned)(quarter * 32) << 16;
    constexpr int HC = BN / 2;                       // keys a thread
    // where the two threads of a row swap values: see attention_tcgen05.cu
    constexpr bool X_SPARE = BN + DV + BN / 2 + 4 <= 256;
    const unsigned x_mine = X_SPARE ? tmem_p + BN / 2 + lane_sel + half * 2 : tmem_s + lane_sel + half * HC;
    const unsigned x_theirs = X_SPARE ? tmem_p + BN / 2 + lane_sel + (half ^ 1) * 2 : tmem_s + lane_sel + (half ^ 1) * HC;
    bool ok = true;
    for (int it = 0; it < ntiles; ++it) {
      const int j0 = (tile_lo + it) * BN;
      ok = __all_sync(0xffffffffu, mbar_wait(s_full, it & 1, err));
      if (!ok) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      float sc[HC];
#pragma unroll
      for (int c0 = 0; c0 < HC; c0 += 32) tmem_ld32(tmem_s + lane_sel + half * HC + c0, (unsigned*)(sc + c0));
      asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
      if (X_SPARE) {                                   // the scores are in registers: the next tile's may come
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncwarp();
        if (lane == 0) mbar_arrive(s_free);
      }
      if (!(j0 >= clear_lo && j0 + BN <= clear_hi)) {
        const unsigned lo_rel = (unsigned)(row_lo - j0 - half * HC), span = (unsigned)(row_hi - row_lo);
#pragma unroll
        for (int j = 0; j < HC; ++j)
          if (!((unsigned)j - lo_rel < span)) sc[j] = -INFINITY;
      }
      float mx0 = fmaxf(sc[0], sc[1]), mx1 = fmaxf(sc[2], sc[3]), mx2 = fmaxf(sc[4], sc[5]), mx3 = fmaxf(sc[6], sc[7]);
#pragma unroll
      for (int j = 8; j < HC; j += 8) {
        mx0 = at_max3(mx0, sc[j], sc[j + 1]); mx1 = at_max3(mx1, sc[j + 2], sc[j + 3]);
        mx2 = at_max3(mx2, sc[j + 4], sc[j + 5]); mx3 = at_max3(mx3, sc[j + 6], sc[j + 7]);
      }
      float mx = fmaxf(fmaxf(mx0, mx1), fmaxf(mx2, mx3)), mx_other;
      ok = pair_exchange(x_mine + (it & 1), x_theirs + (it & 1), &xbar[quarter], it, mx, &mx_other, err);
      if (!ok) break;
      if (!X_SPARE) {                                  // through with the tile's score columns, the exchange's too
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncwarp();
        if (lane == 0) mbar_arrive(s_free);
      }
      mx = fmaxf(mx, mx_other) * scale_log2;
      // the reference point is the row's largest score so far, so that its weight is 1 and has no rounding
      const bool moves = mx > m_ref;
      float corr = 1.0f;
      if (moves) {
        corr = at_ex2(m_ref - mx);
        m_ref = mx;
        l *= corr;
      }
      const float m_safe = (m_ref == -INFINITY) ? 0.f : m_ref;
      unsigned pk[HC / 2];
      const unsigned long long scale2 = at_pack2(scale_log2, scale_log2), shift2 = at_pack2(-m_safe, -m_safe);
      unsigned long long sum01 = at_pack2(0.f, 0.f), sum23 = sum01;
#pragma unroll
      for (int j = 0; j < HC; j += 4) {
        float x0, x1, x2, x3;
        at_unpack2(at_fma2(at_pack2(sc[j], sc[j + 1]), scale2, shift2), x0, x1);
        at_unpack2(at_fma2(at_pack2(sc[j + 2], sc[j + 3]), scale2, shift2), x2, x3);
        const float p0 = at_ex2(x0), p1 = at_ex2(x1), p2 = at_ex2(x2), p3 = at_ex2(x3);
        sum01 = at_add2(sum01, at_pack2(p0, p1));
        sum23 = at_add2(sum23, at_pack2(p2, p3));
        __nv_bfloat162 h0 = __floats2bfloat162_rn(p0, p1), h1 = __floats2bfloat162_rn(p2, p3);
        pk[j / 2] = *(unsigned*)&h0;
        pk[j / 2 + 1] = *(unsigned*)&h1;
      }
      {
        float a0, a1, a2, a3;
        at_unpack2(sum01, a0, a1);
        at_unpack2(sum23, a2, a3);
        l += (a0 + a1) + (a2 + a3);
      }
      // the product of the tile before has to be through: it read P, and it wrote the output that is rescaled here
      if (it > 0) {
        ok = __all_sync(0xffffffffu, mbar_wait(pv_full, (it - 1) & 1, err));
        if (!ok) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        if (__any_sync(0xffffffffu, moves)) {
#pragma unroll
          for (int c0 = 0; c0 < DV / 2; c0 += 32) {
            unsigned v[32];
            tmem_ld32(tmem_o + lane_sel + half * (DV / 2) + c0, v);
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
            for (int j = 0; j < 32; ++j) v[j] = __float_as_uint(__uint_as_float(v[j]) * corr);
            tmem_st32(tmem_o + lane_sel + half * (DV / 2) + c0, v);
          }
          asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
        }
      }
      if constexpr (HC == 64) tmem_st32(tmem_p + lane_sel + half * (HC / 2), pk);
      else tmem_st16(tmem_p + lane_sel + half * (HC / 2), pk);
      // Rows of V that none of this CTA's queries sees (ahead of the window, behind the last query: another query's, or the
      // next sequence's) may hold infinities: cleared before P V is issued, since 0 times infinity is no 0.
      if (j0 < kmin || j0 + BN > kend) {
        ok = __all_sync(0xffffffffu, mbar_wait(&v_full[it % NV], (it / NV) & 1, err));   // V has landed: nothing overwrites the zeros
        if (!ok) break;
        if (r < BN && (j0 + r >= kend || j0 + r < kmin)) {      // thread r: key row r, half a row of every panel
#pragma unroll
          for (int p = 0; p < VP; ++p) {
            uint4* vrow = (uint4*)(sV + (it % NV) * Shape::V_STAGE + p * PANEL + r * 128 + half * 64);
#pragma unroll
            for (int c = 0; c < 4; ++c) vrow[c] = make_uint4(0u, 0u, 0u, 0u);
          }
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // the zeros, before the MMA reads V
      }
      asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(p_full);
    }
    if (ok) ok = __all_sync(0xffffffffu, mbar_wait(pv_full, (ntiles - 1) & 1, err));
    float lother = 0.f;
    if (ok) ok = pair_exchange(x_mine + (ntiles & 1), x_theirs + (ntiles & 1), &xbar[quarter], ntiles, l, &lother, err);
    if (ok) {
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      float lsum = half == 0 ? l + lother : lother + l;
      if (sink) lsum += at_ex2(sink[head] * 1.4426950408889634f - m_ref);
      const float inv = lsum > 0.f ? 1.0f / lsum : 0.f;
      bf16* orow = out + ((size_t)(qs + t0 + r) * heads + head) * DV + half * (DV / 2);
#pragma unroll
      for (int c0 = 0; c0 < DV / 2; c0 += 32) {
        unsigned v[32];
        tmem_ld32(tmem_o + lane_sel + half * (DV / 2) + c0, v);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
        if (r < ntok) {
#pragma unroll
          for (int c = 0; c < 32; c += 8) {
            uint4 w;
            __nv_bfloat162* h = (__nv_bfloat162*)&w;
#pragma unroll
            for (int q = 0; q < 4; ++q)
              h[q] = __floats2bfloat162_rn(__uint_as_float(v[c + 2 * q]) * inv, __uint_as_float(v[c + 2 * q + 1]) * inv);
            *(uint4*)(orow + c0 + c) = w;
          }
        }
      }
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 1) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_s), "r"(256) : "memory");
  }
}

// ---------------------------------------------------------------------------
template <int NQ, int DV>
static int le_launch(const CUtensorMap& mq, const CUtensorMap& mkv, const CUtensorMap& mr, void* out, const int* q_start,
                     const int* seq_lens, int seq_begin, int seq_end, long long tiles, int heads, int rot, int window,
                     float scale, const float* sink, int* err, cudaStream_t stream) {
  static SmemLimit limit;
  if (const int e = limit.allow(latent_expanded_kernel<NQ, DV>, LeShape<NQ, DV>::SMEM)) return e;
  rllm_launch_pdl(latent_expanded_kernel<NQ, DV>, dim3((unsigned)(tiles * heads)), dim3(LE_THREADS), (size_t)LeShape<NQ, DV>::SMEM, stream,
                  mq, mkv, mr, (bf16*)out, q_start, seq_lens, seq_begin, seq_end, heads, rot, window, scale * 1.4426950408889634f,
                  sink, err);
  RLLM_LAUNCH_CHECK();
  return 0;
}

// Sequences seq_begin .. seq_end - 1 of the step, num_tokens tokens in all.  q: num_q_rows tokens of heads x (nope + rot)
// values, rotated, the rows of the sequences' tokens at q_start.  rows [num_rows, row_stride]: the sequences' visible cached
// rows one sequence behind the other, each from the oldest key of its first query rounded down to LE_ALIGN; their shared
// part at kv_rank.  kv [num_rows, heads nope + heads v]: every head's keys, then every head's values.  nope and v 64 or 128,
// rot a multiple of 8 up to 64; out [., heads v]; sink [heads] or null.
RLLM_EXPORT int rllm_latent_expanded_tcgen05(const void* q, int num_q_rows, const void* kv, const void* rows, int num_rows,
                                             int row_stride, int kv_rank, void* out, const int* q_start, const int* seq_lens,
                                             int seq_begin, int seq_end, int num_tokens, int heads, int nope, int rot, int v,
                                             int window, float scale, const float* sink, int* err, cudaStream_t stream) {
  if (seq_end <= seq_begin || num_tokens <= 0) return 0;
  if (heads <= 0 || num_rows <= 0 || kv_rank <= 0 || rot <= 0 || row_stride < kv_rank + rot || window < 0 || !(scale > 0.f) ||
      !err || num_q_rows < num_tokens)
    return RLLM_E_BADARG;
  if (!(nope == 64 || nope == 128) || !(v == 64 || v == 128) || rot % 8 || rot > 64 || kv_rank % 8 || row_stride % 8 ||
      (((uintptr_t)q | (uintptr_t)kv | (uintptr_t)rows | (uintptr_t)out) & 15))
    return RLLM_E_UNSUPPORTED;
  const long long tiles = ((long long)num_tokens + LE_BM - 1) / LE_BM + (seq_end - seq_begin);
  if (tiles * heads > 0x7fffffffLL || (long long)heads * (nope + v) > 0x7fffffffLL) return RLLM_E_UNSUPPORTED;
  CUtensorMap mq, mkv, mr;
  {
    cuuint64_t dims[3] = {(cuuint64_t)(nope + rot), (cuuint64_t)heads, (cuuint64_t)num_q_rows};
    cuuint64_t strides[2] = {(cuuint64_t)(nope + rot) * 2, (cuuint64_t)heads * (nope + rot) * 2};
    cuuint32_t box[3] = {64, 1, LE_BM};
    if (const int rc = at_encode(&mq, 3, q, dims, strides, box)) return rc;
  }
  const int bn = nope == 64 && v == 64 ? 128 : 64;
  {
    cuuint64_t dims[2] = {(cuuint64_t)heads * (nope + v), (cuuint64_t)num_rows};
    cuuint64_t strides[1] = {(cuuint64_t)heads * (nope + v) * 2};
    cuuint32_t box[2] = {64, (cuuint32_t)bn};
    if (const int rc = at_encode(&mkv, 2, kv, dims, strides, box)) return rc;
  }
  {
    cuuint64_t dims[2] = {(cuuint64_t)rot, (cuuint64_t)num_rows};
    cuuint64_t strides[1] = {(cuuint64_t)row_stride * 2};
    cuuint32_t box[2] = {64, (cuuint32_t)bn};
    if (const int rc = at_encode(&mr, 2, (const bf16*)rows + kv_rank, dims, strides, box)) return rc;
  }
#define LE_LAUNCH(NQ_, DV_) return le_launch<NQ_, DV_>(mq, mkv, mr, out, q_start, seq_lens, seq_begin, seq_end, tiles, heads, \
      rot, window, scale, sink, err, stream)
  if (nope == 64) {
    if (v == 64) LE_LAUNCH(2, 64);
    LE_LAUNCH(2, 128);
  }
  if (v == 64) LE_LAUNCH(3, 64);
  LE_LAUNCH(3, 128);
#undef LE_LAUNCH
}
