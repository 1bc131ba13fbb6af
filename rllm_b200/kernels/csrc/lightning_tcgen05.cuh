// The linear-attention recurrence over long bfloat16 portions on the tcgen05 tensor cores, for both forms of
// lightning_walk.cuh (a fixed decay a head; STEPS: step sizes a token).  Chunks of C = 128 tokens, a chunk's start state S_0:
//   states    S_0 of the next chunk = f S_0 + K^T (w * V)             f, w: what is left of a token at the chunk's end
//   outputs   O = diag(u) (Q S_0) + ((Q K^T) * D) V  (+ skip V)       u, D: what is left at token t of the start, of token j
// What is float32 by this design (the weighted values, the start states, the weights (Q K^T) * D) enters a product as value +
// remainder, two bfloat16 numbers; sums are float32.  lightning_mma.cuh does the same in three kernels on mma.sync; there the
// end states go to memory, a chain reads them and writes the start states, and every head's block stages the group's q and k.
//
// states: one CTA a (head, 32 value columns, sequence) walks the sequence's chunks with its part of the state in registers,
//   so that only the start states go to memory, split and laid out as the outputs' kernel wants them in shared memory.  The
//   32 columns' values and remainders are the 64 columns of the B operand, so one chain of products makes both parts.  A
//   chunk costs about 1 us, of which the loads, the products and the factors (a warp or two each) hide behind the arithmetic:
//   with the arithmetic's own warps doing all of it a chunk took 2.1 us, with copies of 16 bytes in place of TMA 2.8.
// outputs: persistent CTAs share out the (chunk, head) pairs, chunk by chunk, so that consecutive pairs of a group keep q, k
//   and Q K^T (in tensor memory) and only bring their values and start state, one to three pairs ahead.  Eight warps make the
//   weights, which pass as the A operand in tensor memory (between two 32s of tokens they are one factor a row times one a
//   column), eight the results of the pair before, which leave by TMA; with the same 16 warps at both one after the other a
//   pair took 5,700 cycles, so 4,500, bound by the instructions of the scheduler whose warps have the chunk's last 32 tokens.
//   A value that is not finite would reach every token of its chunk (0 times infinity): it is staged as zero and its column
//   is set to NaN from its token on.
// Measured, 2,048 tokens: 64 heads of 128 x 64 with steps 122 -> 50 us (states 20), 16 heads of 128 x 128 97 -> 52 us (the
// activations 13, states 19); the results' distance from float64 2.4e-6 -> 2.3e-6 and 8.5e-7 -> 8.3e-7 of their norm.
#pragma once
#include "lightning_walk.cuh"
#include "attention_tcgen05.cuh"
#include "smem_limit.h"

#define LG_CHUNK 128
#define LGS_THREADS 384          // states: 8 warps of arithmetic, one that loads, one that issues products, two for the factors
#define LGO_THREADS 608          // outputs: 8 warps for the weights, 8 for the results, and one each of the latter
#define LG_COLS 32               // value columns a CTA of the states' kernel

__device__ __forceinline__ void lg_tmem_ld16(unsigned taddr, unsigned* r) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                 "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
               : "r"(taddr) : "memory");
}
// lt_step in two parts, so that the load can lie ahead
__device__ __forceinline__ float lg_step_load(const LtSteps& p, int t, int h, int heads) { return p.dt[(size_t)t * heads + h]; }
__device__ __forceinline__ float lg_step(const LtSteps& p, float dt, int h) {
  const float v = dt + p.dt_bias[h];
  return v > 20.f ? v : log1pf(expf(v));
}
// lambda^e for a whole e >= 0 (lambda^0 = 1 also where lambda is 0)
__device__ __forceinline__ float lg_pow(float log2_lam, int e) { return e == 0 ? 1.0f : exp2f((float)e * log2_lam); }
// where 16 bytes `c` of row `r` lie in a tile of 64 columns a panel (128-byte rows, swizzled), panels `panel` bytes apart
__device__ __forceinline__ unsigned lg_at(int r, int c, int panel) {
  return (unsigned)((c >> 3) * panel + r * 128 + (((c & 7) ^ (r & 7)) << 4));
}
// an operand whose rows are the summed index: 64 columns x 8 rows a swizzle atom, 8 rows on 1024 bytes further (stride
// field), 64 columns on a panel further (leading-dimension field)
__device__ __forceinline__ unsigned long long lg_desc_mn(const void* tile, int panel) {
  return (umma_desc(tile) & ~(0x3FFFull << 16)) | ((unsigned long long)(panel >> 4) << 16);
}
__device__ __forceinline__ unsigned lg_pack(float a, float b) {
  const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
  return *(const unsigned*)&h;
}
// two numbers as two pairs of bfloat16: the values and the remainders
__device__ __forceinline__ void lg_split2(float a, float b, unsigned& hi, unsigned& lo) {
  hi = lg_pack(a, b);
  const unsigned long long minus = at_pack2(-1.f, -1.f);
  at_unpack2(at_fma2(at_pack2(__uint_as_float(hi << 16), __uint_as_float(hi & 0xffff0000u)), minus, at_pack2(a, b)), a, b);
  lo = lg_pack(a, b);
}
__device__ __forceinline__ int lg_chunks(int len, int most) { return min((len + LG_CHUNK - 1) / LG_CHUNK, most); }
__device__ __forceinline__ unsigned long long lg_mul2(unsigned long long a, unsigned long long b) {
  unsigned long long d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
// eight activated values of a row, rounded
template <bool STEPS>
__device__ __forceinline__ uint4 lg_act8(const uint4& raw) {
  if (STEPS) return raw;
  float v[8];
  unpack8(raw, v);
#pragma unroll
  for (int x = 0; x < 8; ++x) v[x] = lt_silu(v[x]);
  return make_uint4(lg_pack(v[0], v[1]), lg_pack(v[2], v[3]), lg_pack(v[4], v[5]), lg_pack(v[6], v[7]));
}

// silu of q, k and v for both kernels (every CTA of a head's columns would otherwise activate the head's keys again, and an
// activation is two trips through the special-function unit): rows [heads d | heads d | heads dv] of `act`.  A thread keeps
// its eight columns and walks the rows.
template <int THREADS>
__global__ void __launch_bounds__(THREADS)
lightning_act_kernel(const bf16* q, const bf16* k, const bf16* v, int stride, const int* __restrict__ q_start, int num_seqs,
                     bf16* act, int kn, int vn) {
  pdl_wait_on(q, k, v);                                    // (the projection ahead wrote them)
  pdl_launch();
  const int c = (blockIdx.x * THREADS + threadIdx.x) * 8, width = 2 * kn + vn;
  if (c >= width) return;
  const bf16* src = c < kn ? q + c : c < 2 * kn ? k + (c - kn) : v + (c - 2 * kn);
  const int last = q_start[num_seqs], step = gridDim.y;
  for (int t = q_start[0] + blockIdx.y; t < last; t += 4 * step) {
    uint4 raw[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) if (t + u * step < last) raw[u] = *(const uint4*)(src + (size_t)(t + u * step) * stride);
#pragma unroll
    for (int u = 0; u < 4; ++u) if (t + u * step < last) *(uint4*)(act + (size_t)(t + u * step) * width + c) = lg_act8<false>(raw[u]);
  }
}

// ---------------------------------------------------------------------------
// stages: of a chunk's keys and values in shared memory
template <int D, int DV> struct LgsShape {
  static constexpr int K = 2 * LG_CHUNK * 128, STAGE = K + LG_CHUNK * 128;                 // (D = 64: the keys' second panel is zeros)
  static constexpr int smem(int stages) { return stages * STAGE + 2048; }
};
template <int D, int DV, bool STEPS>
__global__ void __launch_bounds__(LGS_THREADS, 2)
lightning_states_kernel(const __grid_constant__ CUtensorMap map_k, const __grid_constant__ CUtensorMap map_v,
                        const float* __restrict__ decay, LtSteps steps, float* __restrict__ state, unsigned char* __restrict__ work,
                        const int* __restrict__ q_start, const int* __restrict__ slots, int num_slots, int max_chunks,
                        int heads, int stages, int* __restrict__ err) {
  using Shape = LgsShape<D, DV>;
  constexpr int SLICES = DV / LG_COLS;
  extern __shared__ __align__(1024) unsigned char lg_raw[];
  float* fac = (float*)(lg_raw + stages * Shape::STAGE);   // [2][132]: the tokens' weights, and what is left of the start
  unsigned long long* full = (unsigned long long*)(fac + 264);    // [4] loads -> all: a stage is here
  unsigned long long* empty = full + 4;                    // [4] MMA -> loads
  unsigned long long* fac_full = full + 8;                 // [2] factors -> arithmetic
  unsigned long long* ready = full + 10;                   // [2] arithmetic (8 warps) -> MMA: the values are weighted
  unsigned long long* done = full + 12;                    // [2] MMA -> arithmetic, factors
  unsigned* tmem_slot = (unsigned*)(full + 14);
  pdl_wait();
  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
  const int h = blockIdx.x / SLICES, sl = blockIdx.x % SLICES, s = blockIdx.y;
  const int t0 = q_start[s], len = q_start[s + 1] - t0;
  if (len <= 0) return;
  if (tg_smem(lg_raw) & 1023u) {                           // the swizzled tiles need 1024-byte alignment
    if (tid == 0) atomicOr(err, 32);
    return;
  }
  const int chunks = __shfl_sync(0xffffffffu, lg_chunks(len, max_chunks), 0);
  if (tid == 0) {
    for (int i = 0; i < 4; ++i) { mbar_init(&full[i], 1); mbar_init(&empty[i], 1); }
    for (int i = 0; i < 2; ++i) { mbar_init(&fac_full[i], 32); mbar_init(&ready[i], 8); mbar_init(&done[i], 1); }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"((unsigned long long)&map_k) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"((unsigned long long)&map_v) : "memory");
  }
  if (warp == 9) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tg_smem(tmem_slot)), "r"(128) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  if (D == 64) {
    for (int e = tid; e < stages * LG_CHUNK * 8; e += LGS_THREADS)
      *(uint4*)(lg_raw + (e / (LG_CHUNK * 8)) * Shape::STAGE + LG_CHUNK * 128 + e % (LG_CHUNK * 8) * 16) = make_uint4(0u, 0u, 0u, 0u);
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  pdl_launch();                                            // behind the allocation: see pdl_launch
  const unsigned tmem = __shfl_sync(0xffffffffu, *tmem_slot, 0);
  auto wait = [&](unsigned long long* bar, unsigned parity) { return __all_sync(0xffffffffu, mbar_wait(bar, parity, err)) != 0; };

  if (warp == 8) {
    // keys and the 64 value columns that this CTA's are of; rows behind the portion's end are another's (cleared below)
    if (lane == 0) {
      const int kx = (STEPS ? h / steps.per : h) * D, vx = h * DV + sl / 2 * 64;
      int st = 0, phase = 1;
      for (int c = 0; c < chunks; ++c) {
        if (!mbar_wait(&empty[st], phase, err)) break;
        unsigned char* to = lg_raw + st * Shape::STAGE;
        mbar_expect_tx(&full[st], (unsigned)((D / 64 + 1) * LG_CHUNK * 128));
        for (int x = 0; x < D; x += 64) tma_load_2d(to + (x / 64) * LG_CHUNK * 128, &map_k, kx + x, t0 + c * LG_CHUNK, &full[st]);
        tma_load_2d(to + Shape::K, &map_v, vx, t0 + c * LG_CHUNK, &full[st]);
        if (++st == stages) { st = 0; phase ^= 1; }
      }
    }
    __syncwarp();
  } else if (warp == 9) {
    const unsigned idesc = (1u << 4) | (1u << 7) | (1u << 10) | (1u << 15) | (1u << 16) | ((64u >> 3) << 17) | ((128u >> 4) << 24);
    int st = 0;
    for (int c = 0; c < chunks; ++c) {
      if (!wait(&ready[c & 1], (c >> 1) & 1)) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const unsigned long long da = lg_desc_mn(lg_raw + st * Shape::STAGE, LG_CHUNK * 128), db = lg_desc_mn(lg_raw + st * Shape::STAGE + Shape::K, LG_CHUNK * 128);
      if (umma_elect()) {
#pragma unroll
        for (int kk = 0; kk < LG_CHUNK / 16; ++kk)
          umma_bf16(tmem + (c & 1) * 64, da + (unsigned long long)(kk * (2048 >> 4)), db + (unsigned long long)(kk * (2048 >> 4)), idesc, kk != 0);
        umma_commit(&done[c & 1]);
        umma_commit(&empty[st]);
      }
      __syncwarp();
      if (++st == stages) st = 0;
    }
  } else if (warp >= 10) {
    // the weights of every other chunk's tokens, four a lane: sums of the steps behind a token, never differences of sums from the
    // chunk's start, whose last digits would be the weights' error
    const float l2 = STEPS ? 0.f : log2f(decay[h]);
    const float nrate = STEPS ? -expf(steps.a_log[h]) * 1.4426950408889634f : 0.f;
    float next[4];
    auto fetch = [&](int c) {
#pragma unroll
      for (int x = 0; x < 4; ++x) {
        const int t = c * LG_CHUNK + 4 * lane + x;
        next[x] = STEPS && t < len ? lg_step_load(steps, t0 + t, h, heads) : 0.f;
      }
    };
    fetch(warp - 10);
    for (int c = warp - 10; c < chunks; c += 2) {
      const int n = min(LG_CHUNK, len - c * LG_CHUNK);
      float raw[4], w[4], f;
#pragma unroll
      for (int x = 0; x < 4; ++x) raw[x] = next[x];
      fetch(c + 2);
      if (STEPS) {
        float dt[4], after[4];
#pragma unroll
        for (int x = 0; x < 4; ++x) dt[x] = 4 * lane + x < n ? lg_step(steps, raw[x], h) : 0.f;
        after[3] = 0.f;
#pragma unroll
        for (int x = 3; x > 0; --x) after[x - 1] = after[x] + dt[x];
        float sum = after[0] + dt[0];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const float down = __shfl_down_sync(0xffffffffu, sum, o);
          if (lane + o < 32) sum += down;
        }
        f = exp2f(nrate * sum);                            // (lane 0's)
        float later = __shfl_down_sync(0xffffffffu, sum, 1);
        if (lane == 31) later = 0.f;
#pragma unroll
        for (int x = 0; x < 4; ++x) w[x] = exp2f(nrate * (after[x] + later)) * dt[x];
      } else {
#pragma unroll
        for (int x = 0; x < 4; ++x) w[x] = 4 * lane + x < n ? lg_pow(l2, n - 1 - 4 * lane - x) : 0.f;
        f = powf(decay[h], (float)n);
      }
      if (c >= 2 && !wait(&done[c & 1], ((c - 2) >> 1) & 1)) break;                        // the factors of chunk c - 2 are used
      float* to = fac + (c & 1) * 132;
      *(float4*)(to + 4 * lane) = make_float4(w[0], w[1], w[2], w[3]);
      if (lane == 0) to[128] = f;
      mbar_arrive(&fac_full[c & 1]);
    }
  } else {
    // this thread's part of the state: row i, 16 columns
    const int quarter = warp & 3, half = warp >> 2, row = quarter * 32 + lane, col = sl * LG_COLS + half * 16;
    const int slot = slots[s];
    float* sp = (slot >= 0 && slot < num_slots) ? state + (((size_t)slot * heads + h) * D + row) * DV + col : nullptr;
    if (row >= D) sp = nullptr;
    float S[16];
#pragma unroll
    for (int x = 0; x < 16; x += 4) {
      const float4 a = sp ? *(const float4*)(sp + x) : make_float4(0.f, 0.f, 0.f, 0.f);
      S[x] = a.x; S[x + 1] = a.y; S[x + 2] = a.z; S[x + 3] = a.w;
    }
    const unsigned mine = tmem + ((unsigned)(quarter * 32) << 16) + half * 16;
    const bool odd = lane & 1;
    unsigned char* to = work + ((size_t)s * max_chunks * heads + h) * D * DV * 4;
    const unsigned at0 = lg_at(row & ~1, col / 8 + odd, D * 128), at1 = lg_at(row | 1, col / 8 + odd, D * 128);
    // chunk c's start state to memory, then the state at its end; false: a wait ran out
    auto chain = [&](int c, float f) {
      if (quarter * 32 < D) {
        uint4 part[2][2];                                  // [value, remainder][eight columns]
#pragma unroll
        for (int x = 0; x < 8; ++x)
          lg_split2(S[2 * x], S[2 * x + 1], ((unsigned*)&part[0][x >> 2])[x & 3], ((unsigned*)&part[1][x >> 2])[x & 3]);
        // two neighbours swap, so that they write 32 bytes of one row and then of the other
#pragma unroll
        for (int p = 0; p < 2; ++p) {
          const uint4 send = odd ? part[p][0] : part[p][1];
          uint4 got;
          got.x = __shfl_xor_sync(0xffffffffu, send.x, 1); got.y = __shfl_xor_sync(0xffffffffu, send.y, 1);
          got.z = __shfl_xor_sync(0xffffffffu, send.z, 1); got.w = __shfl_xor_sync(0xffffffffu, send.w, 1);
          *(uint4*)(to + p * D * DV * 2 + at0) = odd ? got : part[p][0];
          *(uint4*)(to + p * D * DV * 2 + at1) = odd ? part[p][1] : got;
        }
      }
      to += (size_t)heads * D * DV * 4;
      if (!wait(&done[c & 1], (c >> 1) & 1)) return false;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      unsigned zh[16], zl[16];
      lg_tmem_ld16(mine + (c & 1) * 64, zh);
      lg_tmem_ld16(mine + (c & 1) * 64 + 32, zl);
      asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
      for (int x = 0; x < 16; ++x) S[x] = fmaf(f, S[x], __uint_as_float(zh[x]) + __uint_as_float(zl[x]));
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      return true;
    };
    bool ok = true;
    float f_prev = 0.f;
    int st = 0, phase = 0;
    for (int c = 0; c < chunks; ++c) {
      ok = wait(&full[st], phase) && wait(&fac_full[c & 1], (c >> 1) & 1);
      if (!ok) break;
      unsigned char* sV = lg_raw + st * Shape::STAGE + Shape::K;
      const float* fc = fac + (c & 1) * 132;
      const float f = fc[128];
      const int n = min(LG_CHUNK, len - c * LG_CHUNK);
      // in place: eight of this CTA's columns, in the row's first or second half, become their values and remainders
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const int j = u * 64 + (tid >> 2), c8 = tid & 3;
        const float w = fc[j];
        uint4 hi = *(const uint4*)(sV + lg_at(j, (sl & 1) * 4 + c8, 0)), lo;
        if (j >= n) hi = make_uint4(0u, 0u, 0u, 0u);
        float x[8];
        unpack8(hi, x);
#pragma unroll
        for (int i = 0; i < 4; ++i) lg_split2(x[2 * i] * w, x[2 * i + 1] * w, ((unsigned*)&hi)[i], ((unsigned*)&lo)[i]);
        *(uint4*)(sV + lg_at(j, c8, 0)) = hi;
        *(uint4*)(sV + lg_at(j, c8 + 4, 0)) = lo;
      }
      if (n < LG_CHUNK) {
        for (int e = n * 8 + tid; e < LG_CHUNK * 8; e += 256)
          for (int x = 0; x < D / 64; ++x) *(uint4*)(lg_raw + st * Shape::STAGE + x * LG_CHUNK * 128 + e * 16) = make_uint4(0u, 0u, 0u, 0u);
      }
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(&ready[c & 1]);
      if (c > 0) ok = chain(c - 1, f_prev);
      if (!ok) break;
      f_prev = f;
      if (++st == stages) { st = 0; phase ^= 1; }
    }
    if (ok) ok = chain(chunks - 1, f_prev);
    if (ok && sp) {
#pragma unroll
      for (int x = 0; x < 16; x += 4) *(float4*)(sp + x) = make_float4(S[x], S[x + 1], S[x + 2], S[x + 3]);
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 9) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(128) : "memory");
}

// ---------------------------------------------------------------------------
// The outputs' kernel's values as they have landed, by the 256 threads of its results' warps: zeros behind the chunk's n tokens;
// and as the tile is multiplied by weights that are zero for earlier tokens, a value that is not finite becomes a zero, and
// bad[column] remembers its (first) token with the number of the task, the larger the earlier.
template <int W>
__device__ __noinline__ void lg_make_finite(unsigned char* tile, int n, int tid, int* bad, int* any, int task) {
#pragma unroll 1
  for (int u = 0; u < LG_CHUNK * W / 2048; ++u) {
    const int e = u * 256 + tid, j = e / (W / 8), c = e % (W / 8);
    unsigned* x = (unsigned*)(tile + lg_at(j, c, LG_CHUNK * 128));
#pragma unroll 1
    for (int i = 0; i < 8; ++i) {
      const unsigned bits = 0x7f80u << (16 * (i & 1)), w = x[i >> 1];
      if (j < n && (w & bits) == bits) {
        x[i >> 1] = w & ~(0xffffu << (16 * (i & 1)));
        atomicMax(&bad[c * 8 + i], task << 8 | (255 - j));
        *any = task;
      }
    }
  }
}
template <int W>
__device__ __forceinline__ bool lg_finite(unsigned char* tile, int n, int tid, int* bad, int* any, int task) {
  const unsigned m = 0x7f807f80u, one = 0x00800080u;
  unsigned found = 0u;
#pragma unroll
  for (int u = 0; u < LG_CHUNK * W / 2048; ++u) {
    const int e = u * 256 + tid, j = e / (W / 8);
    uint4* at = (uint4*)(tile + lg_at(j, e % (W / 8), LG_CHUNK * 128));
    const uint4 w = *at;
    if (j >= n) *at = make_uint4(0u, 0u, 0u, 0u);
    else found |= ((w.x & m) + one) | ((w.y & m) + one) | ((w.z & m) + one) | ((w.w & m) + one);
  }
  if (found & 0x80008000u) lg_make_finite<W>(tile, n, tid, bad, any, task);
  return (found & 0x80008000u) != 0u || n < LG_CHUNK;
}

// where a task's chunk is
struct LgPlace { int t0, n, len, s, chunk, h; };

template <int D, int DV> struct LgoShape {
  static constexpr int Q = (D / 64) * 16384, V = (DV / 64) * 16384, S = D * DV * 4;
  static constexpr int NV = DV == 64 ? 3 : 1, NS = DV == 64 ? 2 : 1;                       // stages of values and of start states
  static constexpr int SMEM = 2 * Q + NV * V + NS * S + 32768 + 6656;
};
template <int D, int DV, bool STEPS>
__global__ void __launch_bounds__(LGO_THREADS, 1)
lightning_outputs_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                         const __grid_constant__ CUtensorMap map_v, const __grid_constant__ CUtensorMap map_out,
                         const float* __restrict__ decay, LtSteps steps,
                         const unsigned char* __restrict__ work, const int* __restrict__ q_start, int num_seqs, int max_chunks,
                         float* __restrict__ out, int heads, int* __restrict__ err) {
  using Shape = LgoShape<D, DV>;
  constexpr int NV = Shape::NV, NS = Shape::NS, ND = NS;   // (ND: pairs of results in tensor memory)
  extern __shared__ __align__(1024) unsigned char lg_raw[];
  unsigned char *sQ = lg_raw, *sK = sQ + Shape::Q, *sV = sK + Shape::Q, *sS = sV + NV * Shape::V, *sO = sS + NS * Shape::S;
  // [2] of: log2 of what is left of a token's state since the 32 tokens began [128] | a token's part at the end of its 32
  // [128] | steps [128] | log2 of what the four 32s leave
  float* fac = (float*)(sO + 32768);
  int* bad = (int*)(fac + 1024);                           // [3][DV] where a column stops to be finite, tasks in turn
  int* any = bad + 384;                                    // [3 of 4] the last task that has such a column
  unsigned long long* v_full = (unsigned long long*)(any + 4);    // [3] loads -> results
  unsigned long long* s_full = v_full + 3;                 // [2] loads -> MMA: the start state
  unsigned long long* qk_full = v_full + 5;                // loads -> MMA
  unsigned long long* raw_full = v_full + 6;               // MMA -> weights: Q K^T
  unsigned long long* o_full = v_full + 7;                 // [2] MMA -> all: a task's products
  unsigned long long* v_ready = v_full + 9;                // [2] results (8 warps) -> MMA
  unsigned long long* raw_read = v_full + 11;              // weights (8 warps) -> MMA
  unsigned long long* p_full = v_full + 12;                // weights (8 warps) -> MMA
  unsigned long long* d_free = v_full + 13;                // [3] results (8 warps) -> MMA, loads, factors: through with a task
  unsigned long long* fac_full = v_full + 16;              // [2] factors (32 lanes) -> weights, results
  unsigned* tmem_slot = (unsigned*)(v_full + 18);
  pdl_wait();
  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
  if (tg_smem(lg_raw) & 1023u) {
    if (tid == 0) atomicOr(err, 32);
    return;
  }
  long long total = 0;
  for (int i = 0; i < num_seqs; ++i) total += lg_chunks(q_start[i + 1] - q_start[i], max_chunks);
  total *= heads;
  const int first = __shfl_sync(0xffffffffu, (int)(total * blockIdx.x / gridDim.x), 0);
  const int last = __shfl_sync(0xffffffffu, (int)(total * (blockIdx.x + 1) / gridDim.x), 0), tasks = last - first;
  if (tasks <= 0) return;
  if (tid == 0) {
    for (int i = 0; i < 9; ++i) mbar_init(&v_full[i], 1);
    for (int i = 9; i < 16; ++i) mbar_init(&v_full[i], 8);
    for (int i = 16; i < 18; ++i) mbar_init(&v_full[i], 32);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"((unsigned long long)&map_q) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"((unsigned long long)&map_k) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"((unsigned long long)&map_v) : "memory");
  }
  for (int e = tid; e < 388; e += LGO_THREADS) bad[e] = 0;                                 // (and `any`)
  if (warp == 16) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tg_smem(tmem_slot)), "r"(512) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  pdl_launch();                                            // behind the allocation: see pdl_launch
  // Q K^T: 128 columns, the weights: 128, ND times what the start state gives and what the values give: DV each
  const unsigned tmem_raw = __shfl_sync(0xffffffffu, *tmem_slot, 0), tmem_p = tmem_raw + 128, tmem_d = tmem_raw + 256;
  auto wait = [&](unsigned long long* bar, unsigned parity) { return __all_sync(0xffffffffu, mbar_wait(bar, parity, err)) != 0; };
  // Task m's of barriers that tasks take in turn.  Whoever waits for a phase is needed for the barrier's next one (so that a
  // phase is never two behind, where its parity would look unfinished): three of d_free, for which V waits three tasks late.
  auto wait_task = [&](unsigned long long* bars, int m) { return wait(&bars[m & 1], (m >> 1) & 1); };
  auto wait_free = [&](int m) { return wait(&d_free[m % 3], (m / 3) & 1); };
  LgPlace p;
  p.h = first % heads;
  p.chunk = first / heads;
  for (p.s = 0;; ++p.s) {
    p.t0 = q_start[p.s];
    p.len = q_start[p.s + 1] - p.t0;
    const int n = lg_chunks(p.len, max_chunks);
    if (p.chunk < n) break;
    p.chunk -= n;
  }
  p.n = min(LG_CHUNK, p.len - p.chunk * LG_CHUNK);
  p.t0 += p.chunk * LG_CHUNK;
  // the next task's: the next head, or the first one of the next chunk
  auto advance = [&](LgPlace p) {
    if (++p.h < heads) return p;
    p.h = 0;
    if (p.chunk + 1 < lg_chunks(p.len, max_chunks)) {
      ++p.chunk;
      p.t0 += LG_CHUNK;
    } else {
      p.chunk = 0;
      do {
        ++p.s;
        p.t0 = q_start[p.s];
        p.len = q_start[p.s + 1] - p.t0;
      } while (p.len <= 0);
    }
    p.n = min(LG_CHUNK, p.len - p.chunk * LG_CHUNK);
    return p;
  };
  // q and k are loaded, and Q K^T is made, where the chunk or the group is another than the task's before
  auto fresh = [&](const LgPlace& p, int m) { return m == 0 || !STEPS || p.h % steps.per == 0; };

  if (warp == 18) {
    for (int m = 0; m < tasks; ++m) {
      if (m >= NS && !wait_task(o_full, m - NS)) break;    // the stage's last task has used its start state
      if (lane == 0) {
        const int st = m % NS;
        mbar_expect_tx(&s_full[st], (unsigned)Shape::S);
        asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                     ::"r"(tg_smem(sS + st * Shape::S)), "l"(work + (((size_t)p.s * max_chunks + p.chunk) * heads + p.h) * Shape::S),
                       "r"((unsigned)Shape::S), "r"(tg_smem(&s_full[st])) : "memory");
      }
      __syncwarp();
      if (m >= NV && !wait_free(m - NV)) break;            // the stage's last task is through
      if (lane == 0) {
        const int st = m % NV;
        mbar_expect_tx(&v_full[st], (unsigned)Shape::V);
        for (int x = 0; x < DV; x += 64) tma_load_2d(sV + st * Shape::V + (x / 64) * 16384, &map_v, p.h * DV + x, p.t0, &v_full[st]);
      }
      __syncwarp();
      if (fresh(p, m)) {
        if (m > 0 && !wait_task(o_full, m - 1)) break;     // q's and k's last products are made
        if (lane == 0) {
          const int x0 = (STEPS ? p.h / steps.per : p.h) * D;
          mbar_expect_tx(qk_full, (unsigned)(2 * Shape::Q));
          for (int x = 0; x < D; x += 64) {
            tma_load_2d(sQ + (x / 64) * 16384, &map_q, x0 + x, p.t0, qk_full);
            tma_load_2d(sK + (x / 64) * 16384, &map_k, x0 + x, p.t0, qk_full);
          }
        }
        __syncwarp();
      }
      if (m + 1 < tasks) p = advance(p);
    }
  } else if (warp == 16) {
    const unsigned idesc_qk = (1u << 4) | (1u << 7) | (1u << 10) | ((128u >> 3) << 17) | ((128u >> 4) << 24);
    const unsigned idesc_v = (1u << 4) | (1u << 7) | (1u << 10) | (1u << 16) | ((unsigned)(DV >> 3) << 17) | ((128u >> 4) << 24);
    const unsigned long long dq = umma_desc(sQ), dk = umma_desc(sK);
    int keys = 0;                                          // how many q and k there were
    for (int m = 0; m < tasks; ++m) {
      if (fresh(p, m)) {
        if (!wait(qk_full, keys & 1) || (m > 0 && !wait(raw_read, (m - 1) & 1))) break;
        ++keys;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        if (umma_elect()) {
#pragma unroll
          for (int kk = 0; kk < D / 16; ++kk)
            umma_bf16(tmem_raw, dq + (unsigned long long)((kk >> 2) * (16384 >> 4) + 2 * (kk & 3)),
                      dk + (unsigned long long)((kk >> 2) * (16384 >> 4) + 2 * (kk & 3)), idesc_qk, kk != 0);
          umma_commit(raw_full);
        }
        __syncwarp();
      }
      if (!wait(&s_full[m % NS], (m / NS) & 1) || (m >= ND && !wait_free(m - ND))) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const unsigned tmem_s = tmem_d + m % ND * (2 * DV), tmem_v = tmem_s + DV;
      const unsigned long long ds = lg_desc_mn(sS + m % NS * Shape::S, D * 128);
      if (umma_elect()) {
#pragma unroll
        for (int kk = 0; kk < 2 * (D / 16); ++kk) {
          const int k1 = kk % (D / 16);
          umma_bf16(tmem_s, dq + (unsigned long long)((k1 >> 2) * (16384 >> 4) + 2 * (k1 & 3)),
                    ds + (unsigned long long)((kk >= D / 16 ? (D * DV * 2) >> 4 : 0) + k1 * (2048 >> 4)), idesc_v, kk != 0);
        }
      }
      __syncwarp();
      if (!wait_task(v_ready, m) || !wait(p_full, m & 1)) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const unsigned long long dv = lg_desc_mn(sV + m % NV * Shape::V, 16384);
      if (umma_elect()) {
#pragma unroll
        for (int kk = 0; kk < 16; ++kk)
          umma_bf16_tmem_a(tmem_v, tmem_p + kk * 8, dv + (unsigned long long)((kk & 7) * (2048 >> 4)), idesc_v, kk != 0);
        umma_commit(&o_full[m & 1]);
      }
      __syncwarp();
      if (m + 1 < tasks) p = advance(p);
    }
  } else if (warp == 17) {
    // what is left of a token, four tokens a lane
    float next_raw[4];
    auto fetch = [&](const LgPlace& p) {
#pragma unroll
      for (int x = 0; x < 4; ++x) next_raw[x] = STEPS && 4 * lane + x < p.n ? lg_step_load(steps, p.t0 + 4 * lane + x, p.h, heads) : 0.f;
    };
    fetch(p);
    for (int m = 0; m < tasks; ++m) {
      float pre[4], end[4], dt[4], all = 0.f;
      if (STEPS) {
        const float nrate = -expf(steps.a_log[p.h]) * 1.4426950408889634f;
        float run[4], back[4];
#pragma unroll
        for (int x = 0; x < 4; ++x) dt[x] = 4 * lane + x < p.n ? lg_step(steps, next_raw[x], p.h) : 0.f;
        run[0] = dt[0];
        back[3] = 0.f;
#pragma unroll
        for (int x = 1; x < 4; ++x) {
          run[x] = run[x - 1] + dt[x];
          back[3 - x] = back[4 - x] + dt[4 - x];
        }
        float ahead = run[3], behind = run[3];
#pragma unroll
        for (int o = 1; o < 8; o <<= 1) {                  // over the eight lanes of 32 tokens
          const float up = __shfl_up_sync(0xffffffffu, ahead, o), down = __shfl_down_sync(0xffffffffu, behind, o);
          if ((lane & 7) >= o) ahead += up;
          if ((lane & 7) + o < 8) behind += down;
        }
        all = nrate * ahead;
        const float before = __shfl_up_sync(0xffffffffu, ahead, 1), after = __shfl_down_sync(0xffffffffu, behind, 1);
        ahead = (lane & 7) ? before : 0.f;
        behind = (lane & 7) < 7 ? after : 0.f;
#pragma unroll
        for (int x = 0; x < 4; ++x) {
          pre[x] = nrate * (ahead + run[x]);
          end[x] = exp2f(nrate * (behind + back[x])) * dt[x];
        }
      } else {
        const float l2 = log2f(decay[p.h]);
#pragma unroll
        for (int x = 0; x < 4; ++x) {
          pre[x] = dt[x] = 0.f;                            // (not read)
          end[x] = lg_pow(l2, 31 - ((4 * lane + x) & 31));
        }
      }
      if (m >= 2 && !wait_free(m - 2)) break;              // task m - 2 has used its factors
      float* f = fac + (m & 1) * 512;
      *(float4*)(f + 4 * lane) = make_float4(pre[0], pre[1], pre[2], pre[3]);
      *(float4*)(f + 128 + 4 * lane) = make_float4(end[0], end[1], end[2], end[3]);
      *(float4*)(f + 256 + 4 * lane) = make_float4(dt[0], dt[1], dt[2], dt[3]);
      if ((lane & 7) == 7) f[384 + (lane >> 3)] = all;
      mbar_arrive(&fac_full[m & 1]);
      if (m + 1 < tasks) {
        p = advance(p);
        fetch(p);
      }
    }
  } else if (warp < 8) {
    // the weights of token t and 64 others, as value + remainder, into tensor memory: of those that are later than the warp's
    // tokens nothing, once; the 32 that are its own tokens with their differences
    const int quarter = warp & 3, half = warp >> 2, t = quarter * 32 + lane;
    const unsigned lane_sel = (unsigned)(quarter * 32) << 16;
    for (int b = 2 * half; b < 2 * half + 2; ++b) {
      if (b > quarter) {
        unsigned z[16];
#pragma unroll
        for (int x = 0; x < 16; ++x) z[x] = 0u;
        tmem_st16(tmem_p + lane_sel + b * 16, z);
        tmem_st16(tmem_p + 64 + lane_sel + b * 16, z);
      }
    }
    int keys = 0;
    for (int m = 0; m < tasks; ++m) {
      if (!wait_task(fac_full, m)) break;
      if (fresh(p, m)) {
        if (!wait(raw_full, keys & 1)) break;
        ++keys;
      }
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const float* fc = fac + (m & 1) * 512;
      const float l2 = STEPS ? 0.f : log2f(decay[p.h]);
      const float lt = STEPS ? fc[t] : 0.f;
      // (every warp waits for the task before, also one without weights: it comes back to these barriers only after the others)
      bool through = m == 0;
#pragma unroll 1
      for (int b = 2 * half; b < 2 * half + 2 && b <= quarter; ++b) {
        const int c0 = b * 32;
        float sc[32];
        tmem_ld32(tmem_raw + lane_sel + c0, (unsigned*)sc);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
        if (b < quarter) {
          // since the 32 tokens of the columns ended, times what was left of them there: one factor a row, one a column
          float sum = lt;
          if (STEPS) for (int x = quarter - 1; x > b; --x) sum += fc[384 + x];
          const float since = STEPS ? exp2f(sum) : lg_pow(l2, t - c0 - 31);
          const unsigned long long since2 = at_pack2(since, since);
#pragma unroll
          for (int j = 0; j < 32; j += 4) {
            const float4 e = *(const float4*)(fc + 128 + c0 + j);
            at_unpack2(lg_mul2(at_pack2(sc[j], sc[j + 1]), lg_mul2(since2, at_pack2(e.x, e.y))), sc[j], sc[j + 1]);
            at_unpack2(lg_mul2(at_pack2(sc[j + 2], sc[j + 3]), lg_mul2(since2, at_pack2(e.z, e.w))), sc[j + 2], sc[j + 3]);
          }
        } else {
#pragma unroll
          for (int j = 0; j < 32; j += 4) {
            float w[4];
            if (STEPS) {
              const float4 lj = *(const float4*)(fc + c0 + j), dj = *(const float4*)(fc + 256 + c0 + j);
              w[0] = at_ex2(lt - lj.x) * dj.x; w[1] = at_ex2(lt - lj.y) * dj.y;
              w[2] = at_ex2(lt - lj.z) * dj.z; w[3] = at_ex2(lt - lj.w) * dj.w;
            } else {
#pragma unroll
              for (int x = 0; x < 4; ++x) w[x] = j + x == lane ? 1.f : at_ex2((float)(lane - j - x) * l2);
            }
#pragma unroll
            for (int x = 0; x < 4; ++x) sc[j + x] = j + x > lane ? 0.f : sc[j + x] * w[x];
          }
        }
        unsigned hi[16], lo[16];
#pragma unroll
        for (int j = 0; j < 32; j += 2) lg_split2(sc[j], sc[j + 1], hi[j / 2], lo[j / 2]);
        if (!through && !wait_task(o_full, m - 1)) break;  // the task before has read its weights
        through = true;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        tmem_st16(tmem_p + lane_sel + b * 16, hi);
        tmem_st16(tmem_p + 64 + lane_sel + b * 16, lo);
      }
      if (!through && !wait_task(o_full, m - 1)) break;
      asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(raw_read);
      if (lane == 0) mbar_arrive(p_full);
      if (m + 1 < tasks) p = advance(p);
    }
  } else {
    // the values as they land, and the results: out = u (Q S_0) + weights V + skip v
    const int quarter = warp & 3, half = (warp - 8) >> 2, t = quarter * 32 + lane, id = tid - 256;
    const unsigned lane_sel = (unsigned)(quarter * 32) << 16;
    unsigned char* mine = sO + (warp - 8) * 4096;          // 32 columns of the warp's tokens, so that whole lines are stored
    auto values = [&](const LgPlace& p, int m) {
      if (!wait(&v_full[m % NV], (m / NV) & 1)) return false;
      // (the fence waits for stores on their way: only where there is something to be seen)
      if (__any_sync(0xffffffffu, lg_finite<DV>(sV + m % NV * Shape::V, p.n, id, bad + m % 3 * 128, any + m % 3, m + 1)))
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(&v_ready[m & 1]);
      return true;
    };
    bool ok = values(p, 0);
    for (int m = 0; m < tasks && ok; ++m) {
      const LgPlace next = m + 1 < tasks ? advance(p) : p;
      ok = wait_task(fac_full, m);
      if (!ok) break;
      const float* fc = fac + (m & 1) * 512;
      float sum = STEPS ? fc[t] : 0.f;
      if (STEPS) for (int x = quarter - 1; x >= 0; --x) sum += fc[384 + x];
      const float u = STEPS ? exp2f(sum) : lg_pow(log2f(decay[p.h]), t + 1), skip = STEPS ? steps.skip[p.h] : 0.f;
      if (NV > 1 && m + 1 < tasks) ok = values(next, m + 1);
      ok = ok && wait_task(o_full, m);
      if (!ok) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const unsigned tmem_s = tmem_d + m % ND * (2 * DV), tmem_v = tmem_s + DV;
      const bool holes = *(volatile int*)(any + m % 3) == m + 1;
#pragma unroll 1
      for (int c0 = half * (DV / 2); c0 < (half + 1) * (DV / 2); c0 += 32) {
        float a[32], b[32];
        tmem_ld32(tmem_s + lane_sel + c0, (unsigned*)a);
        tmem_ld32(tmem_v + lane_sel + c0, (unsigned*)b);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
        const unsigned long long u2 = at_pack2(u, u), skip2 = at_pack2(skip, skip);
#pragma unroll
        for (int j = 0; j < 32; j += 8) {
          uint4 x = make_uint4(0u, 0u, 0u, 0u);
          if (STEPS) x = *(const uint4*)(sV + m % NV * Shape::V + lg_at(t, (c0 + j) / 8, 16384));
          const unsigned w[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
          for (int y = 0; y < 4; ++y) {
            unsigned long long o = at_fma2(at_pack2(a[j + 2 * y], a[j + 2 * y + 1]), u2, at_pack2(b[j + 2 * y], b[j + 2 * y + 1]));
            if (STEPS) o = at_fma2(skip2, at_pack2(__uint_as_float(w[y] << 16), __uint_as_float(w[y] & 0xffff0000u)), o);
            at_unpack2(o, a[j + 2 * y], a[j + 2 * y + 1]);
          }
        }
        if (holes) {
#pragma unroll
          for (int j = 0; j < 32; ++j) {
            const int w = bad[m % 3 * 128 + c0 + j];
            if ((w >> 8) == m + 1 && t >= 255 - (w & 255)) a[j] = __int_as_float(0x7fffffff);
          }
        }
        if (c0 + 32 == (half + 1) * (DV / 2)) {            // the last of the task's tensor memory and values that the warp reads
          asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
          __syncwarp();
          if (lane == 0) mbar_arrive(&d_free[m % 3]);
        }
        if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");     // what lay here before is read
        __syncwarp();
#pragma unroll
        for (int j = 0; j < 8; ++j) *(float4*)(mine + lg_at(lane, j, 0)) = make_float4(a[4 * j], a[4 * j + 1], a[4 * j + 2], a[4 * j + 3]);
        if (p.n == LG_CHUNK) {
          asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
          __syncwarp();
          if (lane == 0)
            asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%1, %2}], [%3];\n\tcp.async.bulk.commit_group;"
                         ::"l"((unsigned long long)&map_out), "r"(p.h * DV + c0), "r"(p.t0 + quarter * 32), "r"(tg_smem(mine)) : "memory");
        } else {
          __syncwarp();
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const int row = j * 4 + (lane >> 3), c = lane & 7, tt = quarter * 32 + row;
            const float4 o = *(const float4*)(mine + lg_at(row, c, 0));
            if (tt < p.n) *(float4*)(out + ((size_t)(p.t0 + tt) * heads + p.h) * DV + c0 + c * 4) = o;
          }
          __syncwarp();
        }
      }
      if (NV == 1 && m + 1 < tasks) ok = values(next, m + 1);
      p = next;
    }
    if (lane == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
    __syncwarp();
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 16) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_raw), "r"(512) : "memory");
}

template <int D, int DV, bool STEPS>
static int lg_launch(const bf16* q, const bf16* k, const bf16* v, int rows, int stride, const float* decay, LtSteps steps, float* state,
                     float* work, bf16* act, const int* q_start, const int* slots, int num_slots, int num_seqs, int max_chunks,
                     float* out, int heads, int* err, cudaStream_t stream) {
  const int sms = tg_num_sms();
  const unsigned ctas = (unsigned)(heads * (DV / LG_COLS)) * (unsigned)num_seqs;
  const int stages = ctas <= (unsigned)sms ? 4 : 2;        // (more than one CTA an SM: two of them share it)
  static SmemLimit limit1, limit2;
  if (const int e = limit1.allow(lightning_states_kernel<D, DV, STEPS>, LgsShape<D, DV>::smem(4))) return e;
  if (const int e = limit2.allow(lightning_outputs_kernel<D, DV, STEPS>, LgoShape<D, DV>::SMEM)) return e;
  if constexpr (!STEPS) {
    const int width = heads * (2 * D + DV), gx = (width / 8 + 255) / 256;
    rllm_launch_pdl(lightning_act_kernel<256>, dim3(gx, (sms * 8 + gx - 1) / gx), dim3(256), (size_t)0, stream, q, k, v, stride,
                    q_start, num_seqs, act, heads * D, heads * DV);
    stride = width;
    q = act;
    k = q + heads * D;
    v = k + heads * D;
  }
  CUtensorMap mq, mk, mv, mo;
  {
    tg_encode_fn enc = tg_get_encode();
    if (!enc) return RLLM_E_UNSUPPORTED;
    cuuint64_t dims[2] = {(cuuint64_t)heads * DV, (cuuint64_t)rows}, strides[1] = {(cuuint64_t)heads * DV * 4};
    cuuint32_t box[2] = {32, 32}, estr[2] = {1, 1};
    if (enc(&mo, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, out, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
            CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_NONE, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
      return RLLM_E_BADARG;
  }
  if (const int rc = tg_make_map(&mq, q, rows, (STEPS ? heads / steps.per : heads) * D, stride, LG_CHUNK)) return rc;
  if (const int rc = tg_make_map(&mk, k, rows, (STEPS ? heads / steps.per : heads) * D, stride, LG_CHUNK)) return rc;
  if (const int rc = tg_make_map(&mv, v, rows, heads * DV, stride, LG_CHUNK)) return rc;
  rllm_launch_pdl(lightning_states_kernel<D, DV, STEPS>, dim3(heads * (DV / LG_COLS), num_seqs), dim3(LGS_THREADS),
                  (size_t)LgsShape<D, DV>::smem(stages), stream, mk, mv, decay, steps, state, (unsigned char*)work, q_start,
                  slots, num_slots, max_chunks, heads, stages, err);
  const long long tasks = (long long)num_seqs * max_chunks * heads;
  rllm_launch_pdl(lightning_outputs_kernel<D, DV, STEPS>, dim3((unsigned)(tasks < sms ? tasks : sms)), dim3(LGO_THREADS),
                  (size_t)LgoShape<D, DV>::SMEM, stream, mq, mk, mv, mo, decay, steps, (const unsigned char*)work, q_start, num_seqs,
                  max_chunks, out, heads, err);
  RLLM_LAUNCH_CHECK();
  return 0;
}

// Whether these kernels are faster than the passes of lightning_mma.cuh, for num_seqs sequences of which the longest has
// `chunks` chunks of 128.  The states' kernel takes a chunk after the other, 1 us each, whatever the number of heads; the
// passes take all chunks side by side and are bound by the work.  us there / here:
//   more than six chunks, 2,048 tokens: 4, 8, 12, 24 heads of 128 x 64 with steps 23.6 / 29.7, 29.7 / 31.7, 39.9 / 33.8, 58 / 40;
//     2, 4, 6, 12 of 128 x 128 without 35.8 / 33.8, 35.8 / 35.8, 52 / 38, 79 / 50; 4 of 128 x 128 without beside 8 decoded
//     tokens 38.7 / 31.2, with steps 32.5 / 28.2: those count as sequences too (4 of 64 x 64 are the exception: 22.0 / 24.8)
//   fewer, with steps: 4 heads of 64 x 64, 300, 512, 768 tokens 11.5 / 12.2, 11.7 / 13.2, 12.5 / 14.8; 10 of them 768 15.2 / 15.3;
//     4 of 128 x 64 512, 768 tokens 14.3 / 14.3, 14.7 / 15.6; 2 of 64 x 128 768 14.3 / 16.1, 4 of them 15.9 / 15.7; 1 of
//     128 x 128 768 15.4 / 16.5, 2 of them 16.3 / 15.3
//   without: 4 heads of 64 x 64, 640 tokens 13.7 / 16.0, 768 13.8 / 16.9
static inline bool lg_pays(bool steps, int chunks, int heads, int num_seqs, int d, int dv) {
  const long long work = (long long)heads * num_seqs * d * dv;
  if (chunks > 6) return work >= 5 << 14;
  if (!steps) return !(d == 64 && dv == 64 && chunks >= 5 && work < 6 << 12);
  if (dv == 64 && chunks >= (d == 64 ? 3 : 6)) return work >= 10 << 12;
  return chunks < 4 || work >= 8 << 12;
}

// The kernels where the head's sizes are built and rows start on 16 bytes; -1: not taken.  max_chunks: of LT_CHUNK tokens
// (the start states of half as many chunks lie in `work`).  act (without STEPS): a row of heads (2 d + dv) values a token.
template <bool STEPS>
static int lg_scan(const bf16* q, const bf16* k, const bf16* v, int rows, int stride, const float* decay, LtSteps steps, float* state,
                   float* work, bf16* act, const int* q_start, const int* slots, int num_slots, int num_seqs, int max_chunks,
                   float* out, int heads, int d, int dv, int* err, cudaStream_t stream) {
  static_assert(LG_CHUNK == 2 * LT_CHUNK, "half as many start states as the chunk passes have");
  const uintptr_t at = (uintptr_t)q | (uintptr_t)k | (uintptr_t)v | (uintptr_t)state | (uintptr_t)work | (uintptr_t)act | (uintptr_t)out;
  const int chunks = (max_chunks + 1) / 2;
  if (!(d == 64 || d == 128) || !(dv == 64 || dv == 128) || stride % 8 || (at & 15) || !err || rows <= 0 || (!STEPS && !act)) return -1;
  if ((long long)num_seqs * chunks * heads > 0x3fffffffLL || (long long)heads * 256 > 0x7fffffffLL) return -1;
  if (!lg_pays(STEPS, chunks, heads, num_seqs, d, dv)) return -1;
#define LG_GO(D_, DV_)                                                                                                    \
  if (d == D_ && dv == DV_)                                                                                               \
    return lg_launch<D_, DV_, STEPS>(q, k, v, rows, stride, decay, steps, state, work, act, q_start, slots, num_slots, num_seqs, chunks, \
                                     out, heads, err, stream)
  LG_GO(64, 64); LG_GO(64, 128); LG_GO(128, 64); LG_GO(128, 128);
#undef LG_GO
  return -1;
}
