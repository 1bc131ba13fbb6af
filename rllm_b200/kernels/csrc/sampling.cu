// Sampling over float32 logits [R, V], a cluster of blocks a row, with the reference's
// pipeline (crates/rllm-sampling/src/sampler.rs:62-169): penalties and biases
// (rllm_logit_edits), masks (rllm_logit_mask), then per row: greedy when
// temperature <= 0 or top_k == 1 (:117), else temperature, top-k, top-p, min-p
// (crates/rllm-sampling/src/logits.rs:5-93) and a draw from the softmax of
// what is left (sampler.rs:194-214).
//
// Differences from the reference, on purpose:
//  * the random number of a draw comes from Philox4x32-10 keyed by the
//    request's seed with the index of the generated token as counter, so a
//    request's samples do not depend on the batch it is in (the reference
//    shares one generator between all requests and ignores the request's
//    seed, sampler.rs:37-51, 200-203);
//  * probability mass is summed in 64-bit fixed point (exp(y - max) * 2^40),
//    which is exact and independent of the order of the additions, so neither
//    the top-p cut nor the draw depends on how threads split a row;
//  * greedy ties go to the lowest index (the reference's max_by gives the
//    last, sampler.rs:184-191); top_k keeps the k largest values and their
//    ties (the reference's threshold, logits.rs:26-31, is the (k+1)-th largest,
//    which keeps k+1); top-p keeps all ties of its last value; the draw takes
//    the first index whose running sum exceeds u, so a masked token is never
//    drawn (the reference's `>=` draws index 0 when u is 0, sampler.rs:208).
#include "common.cuh"
#include <math.h>

#define SAMPLE_THREADS 1024
#define FX_ONE 1099511627776.0f  // 2^40

__device__ __forceinline__ unsigned f2key(float f) {
  unsigned b = __float_as_uint(f);
  return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}
__device__ __forceinline__ float key2f(unsigned k) {
  unsigned b = (k & 0x80000000u) ? (k & 0x7fffffffu) : ~k;
  return __uint_as_float(b);
}
__device__ __forceinline__ unsigned long long fx_mass(float y, float mx) {
  return (unsigned long long)(expf(y - mx) * FX_ONE);
}

__device__ void philox4x32_10(unsigned c0, unsigned c1, unsigned c2, unsigned c3, unsigned k0,
                              unsigned k1, unsigned* out) {
  const unsigned M0 = 0xD2511F53u, M1 = 0xCD9E8D57u, W0 = 0x9E3779B9u, W1 = 0xBB67AE85u;
#pragma unroll
  for (int r = 0; r < 10; ++r) {
    const unsigned hi0 = __umulhi(M0, c0), lo0 = M0 * c0;
    const unsigned hi1 = __umulhi(M1, c2), lo1 = M1 * c2;
    const unsigned n0 = hi1 ^ c1 ^ k0, n2 = hi0 ^ c3 ^ k1;
    c0 = n0; c1 = lo1; c2 = n2; c3 = lo0;
    k0 += W0; k1 += W1;
  }
  out[0] = c0; out[1] = c1; out[2] = c2; out[3] = c3;
}

struct ArgMax { float v; int i; };
__device__ __forceinline__ ArgMax argmax_better(ArgMax a, ArgMax b) {
  if (b.v > a.v || (b.v == a.v && b.i < a.i)) return b;
  return a;
}
__device__ ArgMax block_argmax(ArgMax a, ArgMax* sm) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    ArgMax b; b.v = __shfl_xor_sync(0xffffffffu, a.v, o); b.i = __shfl_xor_sync(0xffffffffu, a.i, o);
    a = argmax_better(a, b);
  }
  __syncthreads();
  if (lane == 0) sm[warp] = a;
  __syncthreads();
  ArgMax r = sm[0];
  for (int w = 1; w < (int)(blockDim.x >> 5); ++w) r = argmax_better(r, sm[w]);
  return r;
}

// Radix descent over the 32-bit order keys of a row, 8 bits a pass, from the
// largest value down.  With by_mass false it finds the key of the k-th largest
// element (target = k, every element weighs 1); with by_mass true the key at
// which the mass of the elements >= it first reaches `target`.  Only elements
// with key >= floor_key take part.
__device__ unsigned radix_select(const float* __restrict__ x, int V, float inv_t, float mx,
                                 unsigned floor_key, unsigned long long target, bool by_mass,
                                 unsigned long long* hist, unsigned* sh_prefix,
                                 unsigned long long* sh_cum) {
  unsigned prefix = 0;
  unsigned long long cum = 0;  // weight of elements above the current prefix range
  for (int pass = 0; pass < 4; ++pass) {
    const int shift = 24 - 8 * pass;
    const unsigned himask = pass == 0 ? 0u : (0xffffffffu << (shift + 8));
    for (int b = threadIdx.x; b < 256; b += blockDim.x) hist[b] = 0ull;
    __syncthreads();
    // The keys of a row crowd into a few bins: the lanes of a warp that hit the same bin add their
    // weights up among themselves (two 32-bit sums of the halves of weights below 2^41), and one of
    // them adds the sum to the bin.  Integer sums: the order does not matter.
    const int lane = threadIdx.x & 31;
    const int iters = (V + (int)blockDim.x - 1) / (int)blockDim.x;
    for (int it = 0; it < iters; ++it) {
      const int i = it * (int)blockDim.x + (int)threadIdx.x;
      unsigned long long w = 0;
      unsigned key = 0;
      if (i < V) {
        const float y = x[i] * inv_t;
        key = f2key(y);
        if (!(key < floor_key || (key & himask) != prefix)) w = by_mass ? fx_mass(y, mx) : 1ull;
      }
      const unsigned bin = w ? ((key >> shift) & 0xffu) : 256u + (unsigned)lane;   // lanes without weight stay alone
      const unsigned m = __match_any_sync(0xffffffffu, bin);
      if (w) {
        const unsigned lo = __reduce_add_sync(m, (unsigned)(w & 0xfffffull));
        const unsigned hi = __reduce_add_sync(m, (unsigned)(w >> 20));
        if (lane == __ffs(m) - 1) atomicAdd(&hist[bin], ((unsigned long long)hi << 20) + lo);
      }
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      unsigned long long c = cum;
      int b = 255;
      for (; b > 0; --b) {
        if (c + hist[b] >= target) break;
        c += hist[b];
      }
      *sh_prefix = prefix | ((unsigned)b << shift);
      *sh_cum = c;
    }
    __syncthreads();
    prefix = *sh_prefix;
    cum = *sh_cum;
    __syncthreads();
  }
  return prefix;
}

__global__ void __launch_bounds__(SAMPLE_THREADS)
sample_kernel(const float* __restrict__ logits, int V, int ld, const float* __restrict__ temperature,
              const int* __restrict__ top_k, const float* __restrict__ top_p,
              const float* __restrict__ min_p, const unsigned long long* __restrict__ seeds,
              const long long* __restrict__ gen_index, int* __restrict__ out_tokens) {
  __shared__ ArgMax sm_arg[32];
  __shared__ unsigned long long hist[256];
  __shared__ unsigned long long seg_sum[SAMPLE_THREADS];
  __shared__ unsigned sh_prefix;
  __shared__ unsigned long long sh_cum;
  __shared__ int sh_pick;
  const int r = blockIdx.x;
  const float* x = logits + (size_t)r * ld;
  const float temp = temperature[r];
  const int k = top_k[r];
  const bool greedy = !(temp > 0.f) || k == 1;
  const float inv_t = greedy ? 1.0f : 1.0f / temp;

  ArgMax best; best.v = -INFINITY; best.i = 0x7fffffff;
  for (int i = threadIdx.x; i < V; i += blockDim.x) {
    ArgMax c; c.v = x[i] * inv_t; c.i = i;
    best = argmax_better(best, c);
  }
  best = block_argmax(best, sm_arg);
  if (greedy || best.v == -INFINITY) {
    if (threadIdx.x == 0) out_tokens[r] = best.i == 0x7fffffff ? 0 : best.i;
    return;
  }
  const float mx = best.v;
  unsigned thr_key = 0u;  // keep keys >= thr_key
  if (k > 0 && k < V) {
    const unsigned kk = radix_select(x, V, inv_t, mx, 0u, (unsigned long long)k, false, hist,
                                     &sh_prefix, &sh_cum);
    thr_key = max(thr_key, kk);
  }
  const float p = top_p[r];
  if (p > 0.f && p < 1.f) {
    // mass of what top-k left
    unsigned long long z = 0;
    for (int i = threadIdx.x; i < V; i += blockDim.x) {
      const float y = x[i] * inv_t;
      if (f2key(y) >= thr_key) z += fx_mass(y, mx);
    }
    seg_sum[threadIdx.x] = z;
    __syncthreads();
    if (threadIdx.x == 0) {
      unsigned long long t = 0;
      for (int i = 0; i < (int)blockDim.x; ++i) t += seg_sum[i];
      sh_cum = t;
    }
    __syncthreads();
    const unsigned long long total = sh_cum;
    __syncthreads();
    unsigned long long target = (unsigned long long)((double)total * (double)p);
    if (target < 1ull) target = 1ull;
    const unsigned pk = radix_select(x, V, inv_t, mx, thr_key, target, true, hist, &sh_prefix, &sh_cum);
    thr_key = max(thr_key, pk);
  }
  const float mp = min_p[r];
  if (mp > 0.f) {
    const unsigned mk = f2key(logf(mp) + mx);
    thr_key = max(thr_key, mk);
  }
  // the draw: contiguous segment per thread, exact integer prefix sums
  const int seg = (V + blockDim.x - 1) / blockDim.x;
  const int lo = threadIdx.x * seg, hi = min(V, lo + seg);
  unsigned long long mine = 0;
  for (int i = lo; i < hi; ++i) {
    const float y = x[i] * inv_t;
    if (f2key(y) >= thr_key) mine += fx_mass(y, mx);
  }
  seg_sum[threadIdx.x] = mine;
  __syncthreads();
  if (threadIdx.x == 0) {
    unsigned long long total = 0;
    for (int i = 0; i < (int)blockDim.x; ++i) total += seg_sum[i];
    unsigned w[4];
    const unsigned long long seed = seeds[r];
    const unsigned long long ctr = (unsigned long long)gen_index[r];
    philox4x32_10((unsigned)ctr, (unsigned)(ctr >> 32), 0u, 0u, (unsigned)seed, (unsigned)(seed >> 32), w);
    const unsigned long long u24 = w[0] >> 8;  // u = u24 / 2^24 in [0, 1)
    const unsigned long long thi = __umul64hi(total, u24), tlo = total * u24;
    const unsigned long long target = (thi << 40) | (tlo >> 24);  // floor(total * u)
    unsigned long long c = 0;
    int pick = blockDim.x - 1;
    for (int i = 0; i < (int)blockDim.x; ++i) {
      if (c + seg_sum[i] > target) { pick = i; break; }
      c += seg_sum[i];
    }
    sh_pick = pick;
    sh_cum = target - c;  // what is left to pass inside the picked segment
  }
  __syncthreads();
  if ((int)threadIdx.x == sh_pick) {
    const unsigned long long rest = sh_cum;
    unsigned long long c = 0;
    int tok = -1, last_kept = -1;
    for (int i = lo; i < hi; ++i) {
      const float y = x[i] * inv_t;
      if (f2key(y) < thr_key) continue;
      const unsigned long long w = fx_mass(y, mx);
      if (w) last_kept = i;
      c += w;
      if (c > rest) { tok = i; break; }
    }
    if (tok < 0) tok = last_kept >= 0 ? last_kept : best.i;
    out_tokens[r] = tok;
  }
}

RLLM_EXPORT int rllm_sample_one_cta(const float* logits, int R, int V, int ld, const float* temperature,
                                    const int* top_k, const float* top_p, const float* min_p,
                                    const unsigned long long* seeds, const long long* gen_index,
                                    int* out_tokens, cudaStream_t stream) {
  if (R <= 0) return 0;
  if (V <= 0 || ld < V) return RLLM_E_BADARG;
  sample_kernel<<<R, SAMPLE_THREADS, 0, stream>>>(logits, V, ld, temperature, top_k, top_p, min_p,
                                                  seeds, gen_index, out_tokens);
  RLLM_LAUNCH_CHECK();
  return 0;
}

// Greedy only: out[r] = lowest index of the largest logit of row r.  A row is cut into `split` ranges,
// one CTA each (a vocabulary of 128k in one CTA is all latency); a range's (max, index) goes to
// `partials`, and the CTA that finds itself last for its row (a counter that the kernel leaves at zero)
// takes the best of the ranges.  Ties go to the lowest index at every level, so the cut changes nothing.
__global__ void __launch_bounds__(SAMPLE_THREADS)
argmax_kernel(const float* __restrict__ logits, int V, int ld, int* __restrict__ out_tokens,
              ArgMax* __restrict__ partials, int* __restrict__ counters, int split) {
  __shared__ ArgMax sm_arg[32];
  __shared__ int s_last;
  pdl_wait_on(logits);
  pdl_launch();
  const int r = blockIdx.y, part = blockIdx.x;
  const float* x = logits + (size_t)r * ld;
  const int per = (((V + split - 1) / split) + 3) & ~3;
  const int lo = part * per, hi = min(V, lo + per);
  ArgMax best; best.v = -INFINITY; best.i = 0x7fffffff;
  if ((((uintptr_t)x) & 15) == 0) {
    // lo is a multiple of 4: 16-byte loads, then the tail
    const int n4 = hi > lo ? (hi - lo) >> 2 : 0;
    const float4* x4 = (const float4*)(x + lo);
    for (int i = threadIdx.x; i < n4; i += blockDim.x) {
      const float4 v = x4[i];
      const int j = lo + 4 * i;
      ArgMax c;
      c.v = v.x; c.i = j; best = argmax_better(best, c);
      c.v = v.y; c.i = j + 1; best = argmax_better(best, c);
      c.v = v.z; c.i = j + 2; best = argmax_better(best, c);
      c.v = v.w; c.i = j + 3; best = argmax_better(best, c);
    }
    for (int i = lo + 4 * n4 + threadIdx.x; i < hi; i += blockDim.x) {
      ArgMax c; c.v = x[i]; c.i = i;
      best = argmax_better(best, c);
    }
  } else {
    for (int i = lo + threadIdx.x; i < hi; i += blockDim.x) {
      ArgMax c; c.v = x[i]; c.i = i;
      best = argmax_better(best, c);
    }
  }
  best = block_argmax(best, sm_arg);
  if (split == 1) {
    if (threadIdx.x == 0) out_tokens[r] = best.i == 0x7fffffff ? 0 : best.i;
    return;
  }
  if (threadIdx.x == 0) {
    partials[(size_t)r * split + part] = best;
    asm volatile("fence.acq_rel.gpu;" ::: "memory");
    const int done = atomicAdd(&counters[r], 1);
    s_last = done == split - 1;
    if (s_last) counters[r] = 0;
  }
  __syncthreads();
  if (!s_last || threadIdx.x >= 32) return;
  asm volatile("fence.acq_rel.gpu;" ::: "memory");
  ArgMax a; a.v = -INFINITY; a.i = 0x7fffffff;
  for (int p = threadIdx.x; p < split; p += 32) {
    ArgMax c;
    c.v = __ldcg(&partials[(size_t)r * split + p].v);
    c.i = __ldcg(&partials[(size_t)r * split + p].i);
    a = argmax_better(a, c);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    ArgMax c; c.v = __shfl_xor_sync(0xffffffffu, a.v, o); c.i = __shfl_xor_sync(0xffffffffu, a.i, o);
    a = argmax_better(a, c);
  }
  if (threadIdx.x == 0) out_tokens[r] = a.i == 0x7fffffff ? 0 : a.i;
}

// How a row of V logits is cut for rllm_argmax, and the scratch it needs: R * split (max, index) pairs of
// 8 bytes and R counters that are zero before the call (the kernel leaves them zero).
RLLM_EXPORT int rllm_argmax_split(int V) {
  const int s = (V + 4095) / 4096;
  return s < 1 ? 1 : (s > 64 ? 64 : s);
}

RLLM_EXPORT int rllm_argmax(const float* logits, int R, int V, int ld, int* out_tokens, void* partials,
                            int* counters, cudaStream_t stream) {
  if (R <= 0) return 0;
  if (V <= 0 || ld < V || R > 65535) return RLLM_E_BADARG;
  const int split = rllm_argmax_split(V);
  if (split > 1 && (!partials || !counters)) return RLLM_E_BADARG;
  return (int)rllm_launch_pdl(argmax_kernel, dim3(split, R), dim3(SAMPLE_THREADS), 0, stream, logits, V, ld,
                              out_tokens, (ArgMax*)partials, counters, split);
}

// ---------------------------------------------------------------------------
// The whole draw as one kernel: a cluster of CTAs a row.  Every CTA keeps its range of the row (x / t) in shared memory,
// so the logits are read from memory once; what the CTAs have to know of one another (a range's maximum, the 256 bins
// of a radix pass, a range's mass) they read from each other's shared memory after a cluster barrier, and every CTA
// works the next step out for itself.  The mass is the same exact 64-bit fixed point as in sample_kernel, the target
// the same floor(total * u), the token the first index whose running sum exceeds it: the same token, however the row is
// cut.  What bounds it is the chain of barriers (maximum, mass, two a radix pass) with a few microseconds of work between
// two of them.  Microseconds at 128,256 logits, against the same chain as separate kernels (4 to 14 launches, every one
// reading the logits again): 8 rows, temperature 29 -> 16, top-p 151 -> 39, top-k 130 -> 31, all options 208 -> 50;
// 64 rows 59 -> 41, 465 -> 107, 375 -> 81, 677 -> 127.  Then with the other CTAs' numbers read a lane a CTA, and a list of the
// last keys instead of a third pass, one launch after another: 8 rows 14.7 -> 14.0, 37.4 -> 35.0, 30.5 -> 27.6, 49.4 -> 43.9;
// 64 rows 37.8 -> 36.6, 102.5 -> 96.0, 77.7 -> 71.7, 123.8 -> 108.7; 8 rows of 32,768 9.5 -> 8.4, 26.4 -> 23.2, 25.0 -> 21.5,
// 40.0 -> 34.8.
// ---------------------------------------------------------------------------
#define SC_BINS 2048
#define SC_SELECT_BYTES (SC_BINS * 8 + SC_BINS * 4 + SC_BINS * 8)      // the last term over the CTAs of a row
#define SC_STAGED_MAX (176 * 1024)       // bytes of a range that are kept in shared memory; a longer one is read again
#define SC_CTAS 8                        // the most CTAs of a row
#define SC_CAND 64                       // keys of a range that are listed behind the second pass
#define SC_WORDS_MAX (1 << 18)           // weights of a range that three words of 14 bits and 32 to count them hold

__device__ __forceinline__ unsigned sc_addr(const void* p, int rank) {
  unsigned a = (unsigned)__cvta_generic_to_shared(p), r;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
  return r;
}
__device__ __forceinline__ unsigned long long sc_ld64(const void* p, int rank) {
  unsigned long long v;
  asm volatile("ld.shared::cluster.u64 %0, [%1];" : "=l"(v) : "r"(sc_addr(p, rank)) : "memory");
  return v;
}
__device__ __forceinline__ unsigned sc_ld32(const void* p, int rank) {
  unsigned v;
  asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(v) : "r"(sc_addr(p, rank)) : "memory");
  return v;
}
__device__ __forceinline__ void sc_barrier() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

template <int THREADS>
__global__ void __launch_bounds__(THREADS)
sample_cluster_kernel(const float* logits, int V, int ld, const float* temperature, const int* top_k, const float* top_p,
                      const float* min_p, const unsigned long long* seeds, const long long* gen_index, int* out_tokens,
                      int select, int staged) {
  constexpr int WARPS = THREADS / 32;
  // Dynamic: the range's bins, the third word of the weights' parts, the whole row's bins of this CTA's slice, and the
  // range of the row times 1 / t.  Without top-k and top-p the range alone.
  extern __shared__ __align__(16) unsigned char sc_raw[];
  unsigned long long* const hist = (unsigned long long*)sc_raw;
  unsigned* const third = (unsigned*)(hist + SC_BINS);
  unsigned long long* const slice = (unsigned long long*)(third + SC_BINS);
  float* const ys = (float*)(sc_raw + (select ? SC_BINS * 12 + SC_BINS * 8 / gridDim.x : 0));
  __shared__ ArgMax sm_arg[32];
  __shared__ __align__(8) ArgMax range_best;          // read by the other CTAs as one word of 64 bits
  __shared__ unsigned long long wsum[WARPS], range_sum, slice_sum, sh_cum, sh_weight;
  __shared__ int sh_pick, sh_bin, cand_n;
  __shared__ unsigned long long sh_rest, all_mass[SC_CAND * SC_CTAS];
  __shared__ unsigned cand[SC_CAND], all_cand[SC_CAND * SC_CTAS], cand_top;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int r = blockIdx.y, cs = gridDim.x, rank = blockIdx.x;       // the cluster is the whole x dimension
  pdl_wait_on(logits, temperature, top_k, top_p, min_p, seeds, gen_index);
  pdl_launch();
  const float* x = logits + (size_t)r * ld;
  const float temp = temperature[r];
  const int k = top_k[r];
  const bool greedy = !(temp > 0.f) || k == 1;
  const float inv_t = greedy ? 1.0f : 1.0f / temp;
  const int per = (((V + cs - 1) / cs) + 3) & ~3;
  const int lo = min(V, rank * per), n = min(V, lo + per) - lo;
  x += lo;
  const bool wide = per > SC_WORDS_MAX;
  auto value = [&](int i) { return staged ? ys[i] : x[i] * inv_t; };

  ArgMax best; best.v = -INFINITY; best.i = 0x7fffffff;
  auto take = [&](int i, float y) {
    if (staged) ys[i] = y;
    ArgMax c; c.v = y; c.i = lo + i;
    best = argmax_better(best, c);
  };
  const int n4 = (((uintptr_t)x) & 15) == 0 ? n >> 2 : 0;
  for (int i = tid; i < n4; i += THREADS) {
    const float4 v = ((const float4*)x)[i];
    take(4 * i, v.x * inv_t); take(4 * i + 1, v.y * inv_t); take(4 * i + 2, v.z * inv_t); take(4 * i + 3, v.w * inv_t);
  }
  for (int i = 4 * n4 + tid; i < n; i += THREADS) take(i, x[i] * inv_t);
  best = block_argmax(best, sm_arg);
  if (tid == 0) range_best = best;
  sc_barrier();
  if (cs > 1) {                                       // a lane a range (eight lanes, four times): one trip to the others' memory
    ArgMax b; b.v = -INFINITY; b.i = 0x7fffffff;
    if ((lane & (SC_CTAS - 1)) < cs) {
      const unsigned long long u = sc_ld64(&range_best, lane & (SC_CTAS - 1));
      b.v = __uint_as_float((unsigned)u); b.i = (int)(u >> 32);
    }
#pragma unroll
    for (int o = SC_CTAS / 2; o > 0; o >>= 1) {
      ArgMax c; c.v = __shfl_xor_sync(0xffffffffu, b.v, o); c.i = __shfl_xor_sync(0xffffffffu, b.i, o);
      b = argmax_better(b, c);
    }
    best = argmax_better(best, b);
  }
  if (greedy || best.v == -INFINITY) {
    if (rank == 0 && tid == 0) out_tokens[r] = best.i == 0x7fffffff ? 0 : best.i;
    sc_barrier();                                     // no CTA leaves while another may read its shared memory
    return;
  }
  const float mx = best.v;
  const int slice_bins = SC_BINS / cs;                // rank c adds up the bins c slice_bins ... of all ranges

  // The threshold of radix_select over the whole row: the largest key such that the keys >= it (and >= floor_key) weigh
  // `target` or more; 11, 11 and 10 bits a pass.  by_mass: an element weighs its mass, else 1.  p > 0: the target is p
  // of all the weight that takes part.
  auto descend = [&](unsigned floor_key, bool by_mass, unsigned long long target, float p) -> unsigned {
    unsigned prefix = 0, himask = 0;
    unsigned long long cum = 0, weight = 0;           // what the keys above the prefix weigh, and those of the prefix
    for (int pass = 0; pass < 3; ++pass) {
      const int shift = pass == 0 ? 21 : (pass == 1 ? 10 : 0);
      if (pass == 2 && weight <= SC_CAND * cs * (by_mass ? fx_mass(key2f(prefix | 0x3ffu), mx) : 1ull)) {
        // The keys that share 22 bits with the threshold are few in a row of unlike values: every range lists its own, and
        // every CTA adds them up for itself (a barrier and a look at a few dozen keys instead of a pass over bins with two
        // barriers).  A longer list anywhere: the pass.  (Where they weigh more than the longest lists could, in a row of
        // like values, nothing is listed: 33 rows of 128,256 equal logits with top-k 47 us, 62 with lists that ran over.)
        if (tid == 0) { cand_n = 0; cand_top = 0u; }
        __syncthreads();
        for (int i = tid; i < n; i += THREADS) {
          const unsigned key = f2key(value(i));
          if (key < floor_key || (key & himask) != prefix) continue;
          const int at = atomicAdd(&cand_n, 1);
          if (at < SC_CAND) cand[at] = key;
        }
        sc_barrier();
        const int mine = lane < cs ? (int)sc_ld32(&cand_n, lane) : 0;
        if (!__any_sync(0xffffffffu, mine > SC_CAND)) {
          int total = 0;                                // the lists one behind the other, all of them here
          for (int c = 0; c < cs; ++c) {
            const int m = __shfl_sync(0xffffffffu, mine, c);
            if (tid < m) {
              const unsigned key = sc_ld32(&cand[tid], c);
              all_cand[total + tid] = key;
              all_mass[total + tid] = by_mass ? fx_mass(key2f(key), mx) : 1ull;
            }
            total += m;
          }
          __syncthreads();
          for (int i = tid; i < total; i += THREADS) {
            const unsigned key = all_cand[i];
            unsigned long long w = cum;
            for (int j = 0; j < total; ++j) w += all_cand[j] >= key ? all_mass[j] : 0ull;
            if (w >= target) atomicMax(&cand_top, key);
          }
          __syncthreads();
          return max(cand_top, prefix);                 // (none reaches the target: all of them)
        }
        sc_barrier();                                   // the lists have been looked at everywhere
      }
      // A weight's 41 bits are added up as three words of 14, with native 32-bit atomics; two of the words stand where
      // the bins' sums will.  A range of more than 2^18 weights could run over them: it takes two words and the carry, which
      // an atomic has to come back with.
      unsigned* const w0 = (unsigned*)hist;
      unsigned* const w1 = w0 + SC_BINS;
      for (int b = tid; b < SC_BINS; b += THREADS) w0[b] = w1[b] = third[b] = 0u;
      if (tid == 0) sh_bin = slice_bins - 1;
      __syncthreads();
      for (int i = tid; i < n; i += THREADS) {
        const float y = value(i);
        const unsigned key = f2key(y);
        if (key < floor_key || (key & himask) != prefix) continue;
        const unsigned bin = (key >> shift) & (SC_BINS - 1);
        if (by_mass) {
          const unsigned long long w = fx_mass(y, mx);
          if (w && wide) {
            const unsigned low = (unsigned)w;
            const unsigned carry = atomicAdd(w0 + bin, low) > ~low ? 1u : 0u;
            atomicAdd(w1 + bin, (unsigned)(w >> 32) + carry);
          } else if (w) {
            atomicAdd(w0 + bin, (unsigned)w & 0x3fffu);
            atomicAdd(w1 + bin, (unsigned)(w >> 14) & 0x3fffu);
            atomicAdd(third + bin, (unsigned)(w >> 28));
          }
        } else {
          atomicAdd(w0 + bin, 1u);
        }
      }
      __syncthreads();
      constexpr int PER = SC_BINS / THREADS;
      unsigned long long mine[PER];
#pragma unroll
      for (int q = 0; q < PER; ++q) {
        const int b = tid + q * THREADS;
        mine[q] = ((unsigned long long)third[b] << 28) + ((unsigned long long)w1[b] << (wide ? 32 : 14)) + w0[b];
      }
      __syncthreads();
#pragma unroll
      for (int q = 0; q < PER; ++q) hist[tid + q * THREADS] = mine[q];
      sc_barrier();
      // every CTA adds up one slice of the bins; reading all bins of all ranges instead took 13 us a pass
      unsigned long long all = 0;
      for (int j = tid; j < slice_bins; j += THREADS) {
        unsigned long long v = 0;
#pragma unroll 8
        for (int c = 0; c < cs; ++c) v += sc_ld64(&hist[rank * slice_bins + j], c);
        slice[j] = v;
        all += v;
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) all += __shfl_xor_sync(0xffffffffu, all, o);
      if (lane == 0) wsum[warp] = all;
      __syncthreads();
      if (warp == 0) {
        all = lane < WARPS ? wsum[lane] : 0ull;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) all += __shfl_xor_sync(0xffffffffu, all, o);
        if (lane == 0) slice_sum = all;
      }
      sc_barrier();
      // the slice that the target falls into, from the top; then the bin in it
      const unsigned long long sums = lane < cs ? sc_ld64(&slice_sum, lane) : 0ull;
      if (pass == 0 && p > 0.f) {
        unsigned long long total = 0;
        for (int c = 0; c < cs; ++c) total += __shfl_sync(0xffffffffu, sums, c);
        target = (unsigned long long)((double)total * (double)p);
        if (target < 1ull) target = 1ull;
      }
      int owner = cs - 1;
      for (;; --owner) {
        const unsigned long long v = __shfl_sync(0xffffffffu, sums, owner);
        if (owner == 0 || cum + v >= target) break;
        cum += v;
      }
      // thread t has `per` bins of the slice, from the top; what lies above a bin is the sum of the threads before
      const int per = (slice_bins + THREADS - 1) / THREADS, first = slice_bins - 1 - tid * per;
      unsigned long long own = 0;
      for (int q = 0; q < per; ++q) if (first - q >= 0) own += sc_ld64(&slice[first - q], owner);
      unsigned long long upto = own;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const unsigned long long v = __shfl_up_sync(0xffffffffu, upto, o);
        if (lane >= o) upto += v;
      }
      if (lane == 31) wsum[warp] = upto;
      __syncthreads();
      unsigned long long before = cum + upto - own;
      for (int w = 0; w < warp; ++w) before += wsum[w];
      upto = before;
      unsigned long long last = 0;
      for (int q = 0; q < per && first - q >= 0; ++q) {      // the highest bin that reaches the target; else bin 0
        last = sc_ld64(&slice[first - q], owner);
        upto += last;
        if (upto >= target) { atomicMin(&sh_bin, tid * per + q); break; }
      }
      __syncthreads();
      if (tid == sh_bin / per) {
        for (int q = 0; q < sh_bin % per; ++q) before += sc_ld64(&slice[first - q], owner);
        sh_cum = before;
        sh_weight = last;
      }
      __syncthreads();
      cum = sh_cum;
      weight = sh_weight;
      prefix |= (unsigned)(owner * slice_bins + slice_bins - 1 - sh_bin) << shift;
      himask = 0xffffffffu << shift;
      __syncthreads();
    }
    return prefix;
  };

  unsigned thr_key = 0u;                              // keep keys >= thr_key
  if (select && k > 0 && k < V) thr_key = descend(0u, false, (unsigned long long)k, 0.f);
  const float p = top_p[r];
  if (select && p > 0.f && p < 1.f) thr_key = max(thr_key, descend(thr_key, true, 0ull, p));
  const float mp = min_p[r];
  if (mp > 0.f) thr_key = max(thr_key, f2key(logf(mp) + mx));

  // the draw: a warp has a contiguous part of the range, walked 32 at a time
  const int part = ((n + WARPS - 1) / WARPS + 31) & ~31, a = min(n, warp * part), b = min(n, a + part);
  auto mass = [&](int i) -> unsigned long long {
    const float y = value(i);
    return f2key(y) >= thr_key ? fx_mass(y, mx) : 0ull;
  };
  unsigned long long sum = 0;
  for (int i = a + lane; i < b; i += 32) sum += mass(i);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
  if (lane == 0) wsum[warp] = sum;
  __syncthreads();
  if (warp == 0) {
    unsigned long long t = lane < WARPS ? wsum[lane] : 0ull;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    if (lane == 0) range_sum = t;
  }
  sc_barrier();
  if (warp == 0) {                                    // a lane a range, then a lane a warp's part
    const unsigned long long mine = lane < cs ? sc_ld64(&range_sum, lane) : 0ull;
    unsigned long long upto = mine;
    for (int o = 1; o < cs; o <<= 1) {
      const unsigned long long v = __shfl_up_sync(0xffffffffu, upto, o);
      if (lane >= o) upto += v;
    }
    const unsigned long long total = __shfl_sync(0xffffffffu, upto, cs - 1);
    unsigned w[4];
    const unsigned long long seed = seeds[r];
    const unsigned long long ctr = (unsigned long long)gen_index[r];
    philox4x32_10((unsigned)ctr, (unsigned)(ctr >> 32), 0u, 0u, (unsigned)seed, (unsigned)(seed >> 32), w);
    const unsigned long long u24 = w[0] >> 8;         // u = u24 / 2^24 in [0, 1)
    const unsigned long long thi = __umul64hi(total, u24), tlo = total * u24;
    const unsigned long long target = (thi << 40) | (tlo >> 24);  // floor(total * u)
    // the first range whose running sum exceeds the target, else the last; in it the first warp's part
    const unsigned over = __ballot_sync(0xffffffffu, lane < cs && upto > target);
    const int range = over ? __ffs(over) - 1 : cs - 1;
    const unsigned long long ahead = __shfl_sync(0xffffffffu, upto - mine, range);
    int pick = -1;
    if (range == rank) {
      const unsigned long long part_sum = lane < WARPS ? wsum[lane] : 0ull;
      unsigned long long run = part_sum;
#pragma unroll
      for (int o = 1; o < WARPS; o <<= 1) {
        const unsigned long long v = __shfl_up_sync(0xffffffffu, run, o);
        if (lane >= o) run += v;
      }
      const unsigned past = __ballot_sync(0xffffffffu, lane < WARPS && ahead + run > target);
      pick = past ? __ffs(past) - 1 : WARPS - 1;
      const unsigned long long before = __shfl_sync(0xffffffffu, run - part_sum, pick);
      if (lane == 0) sh_rest = target - ahead - before;     // what is left to pass inside the picked warp's part
    }
    if (lane == 0) sh_pick = pick;
  }
  sc_barrier();                                       // the last read of another CTA's shared memory lies behind this
  if (warp != sh_pick) return;
  unsigned long long c = 0;
  int tok = -1, last_kept = -1;
  for (int i0 = a; i0 < b && tok < 0; i0 += 32) {
    unsigned long long w = i0 + lane < b ? mass(i0 + lane) : 0ull;
    const unsigned kept = __ballot_sync(0xffffffffu, w != 0);
    if (kept) last_kept = lo + i0 + 31 - __clz(kept);
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned long long v = __shfl_up_sync(0xffffffffu, w, o);
      if (lane >= o) w += v;
    }
    const unsigned over = __ballot_sync(0xffffffffu, c + w > sh_rest);
    if (over) tok = lo + i0 + __ffs(over) - 1;
    c += __shfl_sync(0xffffffffu, w, 31);
  }
  if (tok < 0) tok = last_kept >= 0 ? last_kept : best.i;
  if (lane == 0) out_tokens[r] = tok;
}

template <int THREADS>
static int sample_cluster_launch(const float* logits, int R, int V, int ld, const float* temperature, const int* top_k,
                                 const float* top_p, const float* min_p, const unsigned long long* seeds,
                                 const long long* gen_index, int* out_tokens, int select, int cs, cudaStream_t stream) {
  const long long range = (long long)((((V + cs - 1) / cs) + 3) & ~3) * 4;
  // a long range in shared memory leaves an SM one CTA: plain draws of many rows rather read it again
  const int staged = range <= SC_STAGED_MAX && (select || R < 64 || V < 200000) ? 1 : 0;
  static SmemLimit limit;
  if (const int e = limit.allow(sample_cluster_kernel<THREADS>, SC_STAGED_MAX + SC_SELECT_BYTES)) return e;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(cs, R); cfg.blockDim = dim3(THREADS);
  cfg.dynamicSmemBytes = (staged ? (size_t)range : 0) + (select ? SC_BINS * 12 + SC_BINS * 8 / cs : 0); cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = cs; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = rllm_pdl_enabled() ? 2 : 1;
  return (int)cudaLaunchKernelEx(&cfg, sample_cluster_kernel<THREADS>, logits, V, ld, temperature, top_k, top_p, min_p,
                                 seeds, gen_index, out_tokens, select, staged);
}

// The whole pipeline for any mix of rows (greedy, temperature, top-k, top-p, min-p): the same tokens as
// rllm_sample_one_cta.  select 0: top-k and top-p are left out (no row uses them).
RLLM_EXPORT int rllm_sample(const float* logits, int R, int V, int ld, const float* temperature,
                            const int* top_k, const float* top_p, const float* min_p,
                            const unsigned long long* seeds, const long long* gen_index, int* out_tokens,
                            int select, cudaStream_t stream) {
  if (R <= 0) return 0;
  if (V <= 0 || ld < V || R > 65535) return RLLM_E_BADARG;
  int cs = 8;                            // CTAs a row: the portable most; fewer where a row is so short that they hold it at 2,048 each
  while (cs > 1 && (cs / 2) * 2048 >= V) cs /= 2;
  int threads;
  if (select) {
    // While the rows' clusters all fit at one CTA an SM: 1,024 threads (8 rows with top-p: 39 us, 43 with 512); then two
    // CTAs an SM (16 rows: 49 us, 69 with 1,024).
    threads = R <= 14 ? 1024 : 512;
    if (R >= 256 && V <= 16384) cs = 1;  // many short rows: 1,024 x 16,384 with top-p 781 us with eight CTAs a row, 164 with one
  } else {
    // A plain draw has three barriers and little else: the CTAs are as many and as large as the rows need to fill the GPU
    // about once.  us, rows x logits, with 8 CTAs of 512 threads / as chosen: 1,024 x 64 22 / 12 (1 of 256), 512 x 4,096 28 / 15 (1 of
    // 256), 256 x 16,384 62 / 24 and 256 x 32,000 71 / 36 (4 of 256), 256 x 64,000 88 / 61 (8 of 256), 15 x 262,144 31 / 24 and
    // 15 x 524,288 71 / 46 (8 of 1,024), 256 x 262,144 361 / 257 (8 of 512, read twice).
    if (V <= 2048) {
      cs = 1; threads = 256;
    } else if (V <= 8192) {
      cs = R <= 128 ? 4 : (R <= 256 ? 2 : 1); threads = 256;
    } else if (V >= 400000) {
      threads = 1024;
    } else if (R <= 32) {
      threads = V >= 200000 || (V >= 48000 && R <= 15) ? 1024 : 512;
    } else if (V >= 200000) {
      threads = R < 64 ? 1024 : 512;
    } else if (R <= 64) {
      threads = V >= 100000 ? 512 : 256;
    } else {
      if (V < 48000) cs = 4;
      threads = 256;
    }
  }
#define SC_GO(T_) return sample_cluster_launch<T_>(logits, R, V, ld, temperature, top_k, top_p, min_p, seeds, gen_index, out_tokens, select, cs, stream)
  if (threads == 1024) SC_GO(1024);
  if (threads == 512) SC_GO(512);
  SC_GO(256);
#undef SC_GO
}

// ---------------------------------------------------------------------------
// Penalties and biases on single logits.  One entry per (row, distinct token):
// bias is added first (logits.rs:147-154); then the repetition penalty is
// applied `count` times, dividing a positive logit and multiplying any other
// (:95-110, once per occurrence in the context like the reference's loop);
// then frequency * count and, if count > 0, presence are subtracted (:113-144).
// ---------------------------------------------------------------------------
__global__ void logit_edits_kernel(float* __restrict__ logits, int V, int ld, int n,
                                   const int* __restrict__ rows, const int* __restrict__ tokens,
                                   const int* __restrict__ counts, const float* __restrict__ bias,
                                   const float* __restrict__ rep, const float* __restrict__ freq,
                                   const float* __restrict__ pres) {
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= n) return;
  const int r = rows[e], t = tokens[e], c = counts[e];
  if (t < 0 || t >= V) return;
  float* p = logits + (size_t)r * ld + t;
  float v = *p + bias[e];
  const float rp = rep[r];
  if (rp != 1.0f)
    for (int i = 0; i < c; ++i) v = v > 0.f ? v / rp : v * rp;
  if (c > 0) {
    if (freq[r] != 0.f) v -= freq[r] * (float)c;
    if (pres[r] != 0.f) v -= pres[r];
  }
  *p = v;
}

RLLM_EXPORT int rllm_logit_edits(float* logits, int V, int ld, int n, const int* rows,
                                 const int* tokens, const int* counts, const float* bias,
                                 const float* rep, const float* freq, const float* pres,
                                 cudaStream_t stream) {
  if (n <= 0) return 0;
  logit_edits_kernel<<<(n + 255) / 256, 256, 0, stream>>>(logits, V, ld, n, rows, tokens, counts, bias,
                                                          rep, freq, pres);
  RLLM_LAUNCH_CHECK();
  return 0;
}

// Masks.  Row r keeps only the tokens of its sorted list allowed[allowed_start[r]
// .. allowed_start[r+1]) if that list is not empty (logits.rs:157-166); then the
// n_suppress pairs (row, token) are set to -inf (:169-181, :184-191).
__global__ void allowed_mask_kernel(float* __restrict__ logits, int V, int ld,
                                    const int* __restrict__ allowed_start,
                                    const int* __restrict__ allowed) {
  const int r = blockIdx.y;
  const int b = allowed_start[r], e = allowed_start[r + 1];
  if (e <= b) return;
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= V) return;
  int lo = b, hi = e;
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if (allowed[mid] < i) lo = mid + 1; else hi = mid;
  }
  if (!(lo < e && allowed[lo] == i)) logits[(size_t)r * ld + i] = -INFINITY;
}
__global__ void suppress_kernel(float* __restrict__ logits, int V, int ld, int n,
                                const int* __restrict__ rows, const int* __restrict__ tokens) {
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= n) return;
  const int t = tokens[e];
  if (t >= 0 && t < V) logits[(size_t)rows[e] * ld + t] = -INFINITY;
}

RLLM_EXPORT int rllm_logit_mask(float* logits, int R, int V, int ld, const int* allowed_start,
                                const int* allowed, int n_suppress, const int* sup_rows,
                                const int* sup_tokens, cudaStream_t stream) {
  if (R <= 0) return 0;
  if (allowed_start) {
    dim3 grid((V + 255) / 256, R);
    allowed_mask_kernel<<<grid, 256, 0, stream>>>(logits, V, ld, allowed_start, allowed);
    RLLM_LAUNCH_CHECK();
  }
  if (n_suppress > 0) {
    suppress_kernel<<<(n_suppress + 255) / 256, 256, 0, stream>>>(logits, V, ld, n_suppress, sup_rows,
                                                                  sup_tokens);
    RLLM_LAUNCH_CHECK();
  }
  return 0;
}

// ---------------------------------------------------------------------------
// Log-probabilities (natural log) from a row of raw logits, as the reference's sampler reports them
// (crates/rllm-sampling/src/logprobs.rs:5-28: logit - (max + ln sum exp(logit - max)); :34-70: the N
// largest, in descending order).  One CTA a row; the sum is taken in a fixed order (a thread's strided
// elements in index order, then the threads in order), so a row's values do not depend on the batch.
// Ties in the top N: the lower index first (the reference's order among equals is not defined).
// A place for which nothing is left (N beyond the vocabulary, or -inf logits only) gets id -1.
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(SAMPLE_THREADS)
logprobs_kernel(const float* __restrict__ logits, int V, int ld, const int* __restrict__ tokens, int N,
                float* __restrict__ lp, int* __restrict__ top_ids, float* __restrict__ top_lp) {
  __shared__ ArgMax sm_arg[32];
  __shared__ float sm_f[32];
  pdl_wait_on(logits, tokens);
  pdl_launch();
  const int r = blockIdx.x;
  const float* x = logits + (size_t)r * ld;
  ArgMax best; best.v = -INFINITY; best.i = 0x7fffffff;
  for (int i = threadIdx.x; i < V; i += blockDim.x) { ArgMax c; c.v = x[i]; c.i = i; best = argmax_better(best, c); }
  best = block_argmax(best, sm_arg);
  const float mx = best.v;
  float s = 0.f;
  if (mx != -INFINITY)
    for (int i = threadIdx.x; i < V; i += blockDim.x) s += expf(x[i] - mx);
  s = block_sum(s, sm_f);
  const float log_z = mx + logf(s);
  if (threadIdx.x == 0) {
    const int t = tokens[r];
    lp[r] = (mx == -INFINITY || t < 0 || t >= V) ? -INFINITY : x[t] - log_z;
  }
  // the N largest, one pass each: the best element that comes after the last one found
  ArgMax prev; prev.v = INFINITY; prev.i = -1;
  for (int n = 0; n < N; ++n) {
    ArgMax b; b.v = -INFINITY; b.i = 0x7fffffff;
    for (int i = threadIdx.x; i < V; i += blockDim.x) {
      const float v = x[i];
      if (v == -INFINITY) continue;
      if (v < prev.v || (v == prev.v && i > prev.i)) { ArgMax c; c.v = v; c.i = i; b = argmax_better(b, c); }
    }
    b = block_argmax(b, sm_arg);
    const bool none = b.i == 0x7fffffff;
    if (threadIdx.x == 0) {
      top_ids[(size_t)r * N + n] = none ? -1 : b.i;
      top_lp[(size_t)r * N + n] = none ? -INFINITY : b.v - log_z;
    }
    if (none) { prev.v = -INFINITY; prev.i = 0x7fffffff; } else prev = b;
    __syncthreads();
  }
}

// lp [R]: log-probability of tokens[r] in row r; top_ids, top_lp [R, N]: the N likeliest tokens of every row
// and their log-probabilities (N may be 0).
RLLM_EXPORT int rllm_logprobs(const float* logits, int R, int V, int ld, const int* tokens, int N, float* lp,
                              int* top_ids, float* top_lp, cudaStream_t stream) {
  if (R <= 0) return 0;
  if (V <= 0 || ld < V || N < 0 || !tokens || !lp || (N > 0 && (!top_ids || !top_lp))) return RLLM_E_BADARG;
  return (int)rllm_launch_pdl(logprobs_kernel, dim3(R), dim3(SAMPLE_THREADS), 0, stream, logits, V, ld, tokens, N, lp,
                              top_ids, top_lp);
}
