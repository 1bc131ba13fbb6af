// Attention over cached latent rows, prompt portions of bfloat16 on the tcgen05 tensor cores (see latent_attention_mma.cuh
// for what is computed: every head reads the same cached row, a key of dk values whose first dv values are the value).
//
// One CTA per (tile of 128 rows = consecutive (token, head) pairs of a sequence, part of 256 value columns); key tiles of
// 64 at absolute positions.  A tile's keys lie in shared memory as panels of 64 keys x 64 values, and a panel among the
// CTA's value columns serves twice: as the K-major operand of S = Q K^T and, where it lies, as the MN-major operand of
// P V.  Tensor memory: S 64 columns, the output 256, P 32, the exchange 4.  (All 512 value columns of the largest rows at
// once would leave no room for S; two CTAs that each make the scores multiply 1.5 times what one would have to.)
//   six producer warps.  Pages are short (16 rows), and a TMA request a page and panel would be 36 requests a tile of
//   about 70 cycles each; so the rows come by cp.async, eight lanes a row's 128 bytes, into the swizzle that the
//   instructions read, a warp a panel: four warps the value panels, which lie side by side (P V is one instruction over
//   them), two the other panels, through a ring of slots.
//   two warps that issue the products, one S (and tensor memory), one P V: a tile has 36 + 4 of them, and a product costs
//   the warp that issues it more time than the tensor cores.
//   eight softmax warps: two threads a row, as in attention_tcgen05.cu.
// Q takes 147 KB at 576 values, which leaves room for one tile's value panels and six slots.  What bounds it there is a
// cycle: P V gives the value panels back, the next ones come in (about 1,700 cycles), the scores are finished, the softmax
// runs.  Rows of up to 448 values have two sets of value panels.
// Measured against the mma.sync kernel: 2,048 tokens x 16 heads, rows of 576: 625 -> 213 us (8,192 tokens 9.3 -> 2.90 ms,
// 403 TFLOP/s); 8 heads, rows of 288: 188 -> 68 us (8,192: 2.57 -> 0.45 ms, 645 TFLOP/s).  With a reference point that lagged the
// running maximum 205 us, and there: one warp issuing all products 312 us; the panels shared by all producer warps, one panel
// at a time: 410 us; the value panels brought twice, so that the scores need not wait for P V: 205 us (what the copies add is
// what the wait cost).
// Every wait on an mbarrier is bounded (bit 16 of the error word, then wind-down).  No cluster, no multicast.
#include "attention_tcgen05.cuh"

#define LT_BM 128
#define LT_BN 64
#define LT_PANEL 8192                    // 64 keys x 64 values
#define LT_VP 4                          // value panels of a CTA
#define LT_MAX_PANELS 9
#define LT_RING 6                        // slots of the panels that are no values
#define LT_PW 2                          // their producer warps: a slot always has the same one (LT_RING is a multiple)
#define LT_NP (LT_VP + LT_PW)
#define LT_THREADS (32 * (LT_NP + 10))
#define LT_SMEM_MAX (227 * 1024)

static int lt_smem(int panels, int sets) { return 1024 + panels * 16384 + (LT_RING + sets * LT_VP) * LT_PANEL + 512; }

__global__ void __launch_bounds__(LT_THREADS, 1)
latent_tcgen05_kernel(const __grid_constant__ CUtensorMap map_q, bf16* out, const bf16* cache, const int* block_table,
                      int max_blocks, const int* q_start, const int* seq_lens, int seq_begin, int seq_end, int heads, int dk,
                      int dv, int parts, int panels, int sets, int page_size, int num_pages, int window, float scale_log2,
                      const float* sink, int* err) {
  extern __shared__ unsigned char lt_raw[];
  unsigned char* sQ = (unsigned char*)(((uintptr_t)lt_raw + 1023) & ~(uintptr_t)1023);   // panels x [128 rows][64 values]
  unsigned char* sK = sQ + panels * 16384;        // LT_RING x [64 keys][64 values]
  unsigned char* sV = sK + LT_RING * LT_PANEL;    // sets x LT_VP x [64 keys][64 values]
  unsigned long long* bars = (unsigned long long*)(sV + sets * LT_VP * LT_PANEL);
  unsigned long long* q_full = bars;              // TMA -> S
  unsigned long long* k_full = bars + 1;          // [LT_RING] producers -> S
  unsigned long long* k_empty = k_full + LT_RING; // [LT_RING] S -> producers
  unsigned long long* v_full = k_empty + LT_RING; // [2][LT_VP] producers -> S, P V
  unsigned long long* v_empty = v_full + 2 * LT_VP;   // [2] P V -> producers
  unsigned long long* s_full = v_empty + 2;       // S -> softmax
  unsigned long long* p_full = s_full + 1;        // softmax (8 warps) -> P V
  unsigned long long* pv_full = s_full + 2;       // P V -> softmax
  unsigned long long* s_free = s_full + 3;        // softmax (8 warps) -> S
  unsigned long long* xbar = s_full + 4;          // [4] the two warps of a row quarter, one another
  unsigned* tmem_slot = (unsigned*)(xbar + 4);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int part = blockIdx.x % parts;
  int s = -1, tile = 0;
  {
    int left = blockIdx.x / parts;
    for (int i = seq_begin; i < seq_end; ++i) {
      const int n = ((q_start[i + 1] - q_start[i]) * heads + LT_BM - 1) / LT_BM;
      if (left < n) { s = i; tile = n - 1 - left; break; }       // the rows that see the most keys first
      left -= n;
    }
  }
  if (s < 0) return;
  const int qs = q_start[s], qlen = q_start[s + 1] - qs;
  const int pos0 = seq_lens[s] - qlen;
  const int row0 = tile * LT_BM, rows = min(LT_BM, qlen * heads - row0);      // among the sequence's qlen * heads rows
  const int first_pos = pos0 + row0 / heads, last_pos = pos0 + (row0 + rows - 1) / heads;
  auto oldest = [&](int p) { return (window > 0 && p - window + 1 > 0) ? p - window + 1 : 0; };
  const int kmin = oldest(first_pos), kend = last_pos + 1;
  const int tile_lo = kmin / LT_BN, ntiles = (kend + LT_BN - 1) / LT_BN - tile_lo;
  const int v0 = part * LT_VP, vp = min(LT_VP, (dv + 63) / 64 - v0);          // this CTA's value panels
  const int plain = panels - vp;                                              // the others come first

  if (threadIdx.x == 0) {
    mbar_init(q_full, 1);
    for (int i = 0; i < LT_RING; ++i) { mbar_init(&k_full[i], 1); mbar_init(&k_empty[i], 1); }
    for (int i = 0; i < 2 * LT_VP; ++i) mbar_init(&v_full[i], 1);
    for (int i = 0; i < 2; ++i) mbar_init(&v_empty[i], 1);
    mbar_init(s_full, 1);
    mbar_init(p_full, 8);
    mbar_init(pv_full, 1);
    mbar_init(s_free, 8);
    for (int i = 0; i < 4; ++i) mbar_init(&xbar[i], 2);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"((unsigned long long)&map_q) : "memory");
  }
  if (warp == LT_NP) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tg_smem(tmem_slot)), "r"(512) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const unsigned tmem_s = *tmem_slot, tmem_o = tmem_s + LT_BN, tmem_p = tmem_o + 64 * LT_VP;

  if (warp < LT_NP) {
    if (threadIdx.x == 0) {
      mbar_expect_tx(q_full, (unsigned)(panels * 16384));
      for (int pn = 0; pn < panels; ++pn) tma_load_2d(sQ + pn * 16384, &map_q, pn * 64, qs * heads + row0, q_full);
    }
    __syncwarp();
    // lane l brings chunk l % 8 of the rows l / 8, l / 8 + 4, ... of a panel
    const int chunk = lane & 7, g = lane >> 3;
    const int* bt = block_table + (size_t)s * max_blocks;
    int page[2];                                  // of rows lane and lane + 32; -2 behind the last visible key
    auto fetch = [&](int it) {
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const int j = (tile_lo + it) * LT_BN + lane + 32 * i;
        page[i] = it < ntiles && j < kend ? bt[j / page_size] : -2;
      }
    };
    int at[2];                                    // the rows' places in the cache; -1: zeros (also for rows that the window
                                                  // hides from all of this CTA's queries: 0 times infinity is no 0)
    auto find = [&](int it) {
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const int j = (tile_lo + it) * LT_BN + lane + 32 * i;
        at[i] = page[i] >= 0 && page[i] < num_pages && j >= kmin ? page[i] * page_size + j % page_size : -1;
        if (at[i] < 0 && page[i] != -2 && j >= kmin) atomicOr(err, 4);   // a visible key without a page
      }
    };
    auto ask = [&](unsigned char* to, int panel) {
      const int col = panel * 64 + chunk * 8;
      const bool inside = col < dk;
      const unsigned dst = tg_smem(to) + g * 128;
#pragma unroll
      for (int i = 0; i < 16; ++i) {              // row g + 4 i: its chunks change places by the row's last three bits
        const int row = __shfl_sync(0xffffffffu, at[i >> 3], (g + 4 * i) & 31);
        const int b = row >= 0 && inside ? 16 : 0;
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;"
                     ::"r"(dst + i * 512 + ((chunk ^ ((g + 4 * i) & 7)) << 4)), "l"(b ? cache + (size_t)row * dk + col : cache), "r"(b) : "memory");
      }
      asm volatile("cp.async.commit_group;" ::: "memory");
    };
    // The tensor cores read a panel through the async proxy.  The fence waits for every copy this warp has under way, so a
    // warp has one panel at a time, and the warps are what keeps several on their way.
    auto hand_over = [&](unsigned long long* full) {
      asm volatile("cp.async.wait_group 0;" ::: "memory");
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(full);
    };
    if (warp < LT_VP) {
      if (warp < vp) {
        fetch(0);
        for (int it = 0; it < ntiles; ++it) {
          find(it);
          const int set = sets == 2 ? it & 1 : 0, use = sets == 2 ? it >> 1 : it;
          if (!__all_sync(0xffffffffu, mbar_wait(&v_empty[set], (use & 1) ^ 1, err))) break;
          ask(sV + (set * LT_VP + warp) * LT_PANEL, v0 + warp);
          fetch(it + 1);                          // on its way meanwhile
          hand_over(&v_full[set * LT_VP + warp]);
        }
      }
    } else {
      // panel o of tile it is the n-th of the ring: slot n % LT_RING, warp n % LT_PW
      int it = 0, o = warp - LT_VP, slot = o;
      unsigned phase = 1;
      while (plain > 0 && o >= plain) { o -= plain; ++it; }
      if (plain > 0) fetch(it);
      while (plain > 0 && it < ntiles) {
        find(it);
        if (!__all_sync(0xffffffffu, mbar_wait(&k_empty[slot], phase, err))) break;
        ask(sK + slot * LT_PANEL, o < v0 ? o : o + vp);
        const int here = slot;
        o += LT_PW;
        while (o >= plain) { o -= plain; ++it; }
        slot += LT_PW;
        if (slot >= LT_RING) { slot -= LT_RING; phase ^= 1; }
        fetch(it);
        hand_over(&k_full[here]);
      }
    }
  } else if (warp == LT_NP) {
    // ---- S = Q K^T: the panels that are no values, then the value panels.  The whole warp walks, one lane issues.
    const unsigned idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((unsigned)(LT_BN >> 3) << 17) | ((unsigned)(LT_BM >> 4) << 24);
    const unsigned long long dq = umma_desc(sQ), dk0 = umma_desc(sK), dv0 = umma_desc(sV);
    int slot = 0;
    unsigned phase = 0;
    bool ok = __all_sync(0xffffffffu, mbar_wait(q_full, 0, err));
    for (int it = 0; it < ntiles && ok; ++it) {
      if (it > 0) {                                 // the softmax warps hold the scores of the tile before
        ok = __all_sync(0xffffffffu, mbar_wait(s_free, (it - 1) & 1, err));
        if (!ok) break;
      }
      for (int o = 0; o < plain; ++o) {
        ok = __all_sync(0xffffffffu, mbar_wait(&k_full[slot], phase, err));
        if (!ok) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const unsigned long long a = dq + (unsigned long long)((o < v0 ? o : o + vp) * (16384 >> 4));
        const unsigned long long b = dk0 + (unsigned long long)(slot * (LT_PANEL >> 4));
        if (umma_elect()) {
#pragma unroll
          for (int k = 0; k < 4; ++k) umma_bf16(tmem_s, a + 2 * k, b + 2 * k, idesc, (o | k) != 0);
          umma_commit(&k_empty[slot]);
        }
        __syncwarp();
        if (++slot == LT_RING) { slot = 0; phase ^= 1; }
      }
      if (!ok) break;
      const int set = sets == 2 ? it & 1 : 0, use = sets == 2 ? it >> 1 : it;
      // the value panels come in together: one wait for all of them, then their products in one go
      for (int p = 0; p < vp && ok; ++p) ok = __all_sync(0xffffffffu, mbar_wait(&v_full[set * LT_VP + p], use & 1, err));
      if (!ok) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      unsigned long long a = dq + (unsigned long long)(v0 * (16384 >> 4));
      unsigned long long b = dv0 + (unsigned long long)(set * (LT_VP * LT_PANEL >> 4));
      if (umma_elect()) {
        for (int p = 0; p < vp; ++p) {
#pragma unroll
          for (int k = 0; k < 4; ++k) umma_bf16(tmem_s, a + 2 * k, b + 2 * k, idesc, (plain | p | k) != 0);
          a += 16384 >> 4;
          b += LT_PANEL >> 4;
        }
        umma_commit(s_full);
      }
      __syncwarp();
    }
  } else if (warp == LT_NP + 1) {
    // ---- P V.  V is the MN-major operand: 8 keys on 1024 bytes further (stride field), 64 values on a panel further
    const unsigned idesc = (1u << 4) | (1u << 7) | (1u << 10) | (1u << 16) | ((unsigned)(vp * 8) << 17) | ((unsigned)(LT_BM >> 4) << 24);
    const unsigned long long dv0 = (umma_desc(sV) & ~(0x3FFFull << 16)) | ((unsigned long long)(LT_PANEL >> 4) << 16);
    bool ok = true;
    for (int it = 0; it < ntiles && ok; ++it) {
      const int set = sets == 2 ? it & 1 : 0, use = sets == 2 ? it >> 1 : it;
      for (int p = 0; p < vp && ok; ++p) ok = __all_sync(0xffffffffu, mbar_wait(&v_full[set * LT_VP + p], use & 1, err));
      if (ok) ok = __all_sync(0xffffffffu, mbar_wait(p_full, it & 1, err));        // P is there, O is rescaled
      if (!ok) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const unsigned long long b = dv0 + (unsigned long long)(set * (LT_VP * LT_PANEL >> 4));
      if (umma_elect()) {
#pragma unroll
        for (int kk = 0; kk < LT_BN / 16; ++kk)
          umma_bf16_tmem_a(tmem_o, tmem_p + kk * 8, b + (unsigned long long)(kk * (2048 >> 4)), idesc, (it | kk) != 0);
        umma_commit(&v_empty[set]);
        umma_commit(pv_full);
      }
      __syncwarp();
    }
  } else {
    // ---- softmax: two threads a row; warp w and w + 4 own the same 32 rows
    const int quarter = warp & 3, half = (warp - LT_NP - 2) >> 2;
    const int r = quarter * 32 + lane;
    const bool live = r < rows;
    const int row = row0 + min(r, rows - 1), head = row % heads;
    const int pos = pos0 + row / heads;
    const int row_hi = pos + 1, row_lo = oldest(pos);
    const int clear_lo = oldest(last_pos), clear_hi = first_pos + 1;   // tiles inside need no mask
    float m_ref = -INFINITY, l = 0.f;
    const unsigned lane_sel = (unsigned)(quarter * 32) << 16;
    constexpr int HC = LT_BN / 2;                    // keys a thread
    const unsigned x_mine = tmem_p + LT_BN / 2 + lane_sel + half * 2, x_theirs = tmem_p + LT_BN / 2 + lane_sel + (half ^ 1) * 2;
    const int oc = half * vp * 32;                   // this thread's output columns: vp * 32 from here
    bool ok = true;
    for (int it = 0; it < ntiles; ++it) {
      const int j0 = (tile_lo + it) * LT_BN;
      ok = __all_sync(0xffffffffu, mbar_wait(s_full, it & 1, err));
      if (!ok) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      float sc[HC];
      tmem_ld32(tmem_s + lane_sel + half * HC, (unsigned*)sc);
      asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(s_free);            // the scores are in registers: the next tile's may come
      if (!(j0 >= clear_lo && j0 + LT_BN <= clear_hi)) {
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
      mx = fmaxf(mx, mx_other) * scale_log2;
      // The reference point is the row's largest score so far, so that its weight is 1 and has no rounding.  (Moved only when the
      // max has grown by 2^8, as in attention_tcgen05.cu, results are further from float64 than the mma.sync kernel's.)
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
          for (int c0 = 0; c0 < vp * 32; c0 += 32) {
            unsigned v[32];
            tmem_ld32(tmem_o + lane_sel + oc + c0, v);
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
            for (int j = 0; j < 32; ++j) v[j] = __float_as_uint(__uint_as_float(v[j]) * corr);
            tmem_st32(tmem_o + lane_sel + oc + c0, v);
          }
          asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
        }
      }
      tmem_st16(tmem_p + lane_sel + half * (HC / 2), pk);
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
      bf16* orow = out + ((size_t)qs * heads + row) * dv + v0 * 64;
      for (int c0 = 0; c0 < vp * 32; c0 += 32) {
        const int col = oc + c0;
        unsigned v[32];
        tmem_ld32(tmem_o + lane_sel + col, v);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
        if (live) {
#pragma unroll
          for (int c = 0; c < 32; c += 8) {
            if (v0 * 64 + col + c + 8 <= dv) {         // dv is a multiple of 8
              uint4 w;
              __nv_bfloat162* h = (__nv_bfloat162*)&w;
#pragma unroll
              for (int q = 0; q < 4; ++q)
                h[q] = __floats2bfloat162_rn(__uint_as_float(v[c + 2 * q]) * inv, __uint_as_float(v[c + 2 * q + 1]) * inv);
              *(uint4*)(orow + col + c) = w;
            }
          }
        }
      }
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == LT_NP) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_s), "r"(512) : "memory");
  }
}

// Sequences seq_begin .. seq_end - 1 of the step, num_tokens tokens in all.  q: num_q_rows tokens of heads * dk values,
// the rows of the sequences' tokens at q_start; cache [pages, 1, page_size, dk]; out [., heads * dv].  dk and dv multiples
// of 8, dk up to 576, dv up to 512 and dk; sink [heads] or null.
RLLM_EXPORT int rllm_latent_attention_tcgen05(const void* q, int num_q_rows, void* out, const void* cache,
                                              const int* block_table, int max_blocks, const int* q_start,
                                              const int* seq_lens, int seq_begin, int seq_end, int num_tokens, int heads,
                                              int dk, int dv, int page_size, int num_pages, int window, float scale,
                                              const float* sink, int* err, cudaStream_t stream) {
  if (seq_end <= seq_begin || num_tokens <= 0) return 0;
  if (heads <= 0 || dk <= 0 || dv <= 0 || dv > dk || page_size <= 0 || num_pages <= 0 || max_blocks <= 0 || window < 0 ||
      !(scale > 0.f) || !err || num_q_rows < num_tokens)
    return RLLM_E_BADARG;
  if (dk % 8 || dv % 8 || dk > 64 * LT_MAX_PANELS || dv > 512 || (((uintptr_t)q | (uintptr_t)out | (uintptr_t)cache) & 15) ||
      (long long)num_q_rows * heads > 0x3fffffffLL)
    return RLLM_E_UNSUPPORTED;
  CUtensorMap mq;
  int rc = tg_make_map(&mq, q, num_q_rows * heads, dk, dk, LT_BM);
  if (rc) return rc;
  const int panels = (dk + 63) / 64, parts = (dv + 64 * LT_VP - 1) / (64 * LT_VP);
  const int sets = lt_smem(panels, 2) <= LT_SMEM_MAX ? 2 : 1, smem = lt_smem(panels, sets);
  static SmemLimit limit;
  if (const int e = limit.allow(latent_tcgen05_kernel, LT_SMEM_MAX)) return e;
  const long long tiles = (((long long)num_tokens * heads + LT_BM - 1) / LT_BM + (seq_end - seq_begin)) * parts;
  if (tiles > 0x7fffffffLL) return RLLM_E_UNSUPPORTED;
  latent_tcgen05_kernel<<<dim3((unsigned)tiles), LT_THREADS, smem, stream>>>(
      mq, (bf16*)out, (const bf16*)cache, block_table, max_blocks, q_start, seq_lens, seq_begin, seq_end, heads, dk, dv, parts,
      panels, sets, page_size, num_pages, window, scale * 1.4426950408889634f, sink, err);
  RLLM_LAUNCH_CHECK();
  return 0;
}
