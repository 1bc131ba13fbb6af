// Paged causal attention on CUDA cores, for float32 and bfloat16 caches: the
// kernel of the true 32-bit path, and the fallback of the bfloat16 path for
// shapes its tensor-core kernels refuse.  One warp per (query token, query
// head), or a block of eight where there are few of them; it serves prompt
// portions and single decoded tokens alike, since a token's keys are read from
// the cache through the block table either way.
//
// Contract (the reference's intended one, crates/rllm-kernels/src/cuda/
// paged_attention.cu:88-179 for the math; its prefill kernel ignores earlier
// context at :285-286, which this does not): the query at position p of
// sequence s sees keys max(0, p - window + 1) .. p of s (window 0: all keys
// 0 .. p); kv head of query head h is h / (nq / nkv) (:113); scores are
// scaled by `scale`; softmax is online in float32 (:159-169), P.V is
// accumulated in float32 and divided by the sum once (:173-178).
//
// Options beyond that contract (each off at 0 / null):
//   keep_first  with a window: keys 0 .. keep_first - 1 stay visible however far back they lie;
//   chunk       the query sees only keys of its own chunk, floor(j / chunk) == floor(p / chunk);
//   softcap     score <- softcap * tanh(score / softcap) after the scaling;
//   sinks       float32 [nq]: exp(sinks[h]) joins the softmax's denominator (no key, no value, unscaled);
//   gate        a row of gate pre-activations beside the token's queries: the result is multiplied by
//               sigmoid(gate[h]) (gate_mode 1, one number a head) or sigmoid(gate[h * dv + i])
//               (gate_mode 2, one a result element);
//   slopes      float32 [nq]: slopes[h] * (p - j) is taken off the score of key j (after scaling and cap):
//               a bias that grows with the distance between query and key.
//
// Keys are walked in groups of 32 aligned to absolute positions; four groups
// (128 keys at absolute positions) make a partial result from an empty start,
// and a row's partial results are added up in order.  So the arithmetic of a
// row does not depend on how the sequence was cut into steps, on the batch
// around it, on which pages hold it, or on how many warps share it.
//
// What bounds it is latency: a lane's key and the 32 values of a group are loads
// that wait for nothing but the block table, so eight keys' worth of values (four
// for heads above 64, two above 128) and up to eight pieces of a key are kept on
// their way.  Four sequences of 100 to 3,000 keys, one token each, 32 heads of 64 in
// float32: 1,225 us with a warp a row and a load at a time, 616 with loads ahead, 92
// with eight warps a row; 6,400 rows of up to 300 keys 264 -> 183.
#include "common.cuh"
#include <math.h>

#define ATT_WARPS 4
#define ATT_MAX_D 256

template <typename T> struct Vec8;
template <> struct Vec8<float> {
  static __device__ __forceinline__ void load(const float* p, float* o) {
    float4 a = *(const float4*)p, b = *(const float4*)(p + 4);
    o[0] = a.x; o[1] = a.y; o[2] = a.z; o[3] = a.w; o[4] = b.x; o[5] = b.y; o[6] = b.z; o[7] = b.w;
  }
};
template <> struct Vec8<bf16> {
  static __device__ __forceinline__ void load(const bf16* p, float* o) {
    uint4 a = *(const uint4*)p;
    const __nv_bfloat162* h = (const __nv_bfloat162*)&a;
#pragma unroll
    for (int i = 0; i < 4; ++i) { float2 f = __bfloat1622float2(h[i]); o[2 * i] = f.x; o[2 * i + 1] = f.y; }
  }
};

#define ATT_PART 128         // keys of a partial result
#define ATT_RESULT(RD) (32 * (RD) + 3)   // its floats: weighted values, largest score, sum of weights, whether NaN was passed over

// d: the size of a query and key head; dv: of a value and output head (they may differ), up to 32 RD.  VEC: d is a
// multiple of 8 and keys are fetched eight at a time; otherwise one by one.  WPR warps share a row.
template <typename T, bool VEC, int RD, int WPR>
__global__ void __launch_bounds__(32 * (WPR == 1 ? ATT_WARPS : WPR), WPR == 1 ? (RD == 2 ? 6 : 8) : 4)
attention_simt_kernel(const T* __restrict__ q, int q_stride, T* __restrict__ out,
                      const T* __restrict__ kcache, const T* __restrict__ vcache,
                      const int* __restrict__ block_table, int max_blocks,
                      const int* __restrict__ positions, const int* __restrict__ token_seq, int T_tokens,
                      int nq, int nkv, int d, int dv, int page_size, int num_pages, int window, float scale,
                      int keep_first, int chunk, float softcap, const float* __restrict__ sinks,
                      const T* __restrict__ gate, int gate_stride, int gate_mode,
                      const float* __restrict__ slopes, int shared_keys, int v_ld, int* __restrict__ err) {
  // keys whose values are on their way together, and pieces of a key.  More of them, or more registers than the bounds above
  // leave (64; 80 for one warp a row and heads up to 64), cost warps in flight: with 87 to 93 registers heads of 256 took 1.5 to
  // 1.9 times as long at 4,096 rows as a load at a time did, 0.97 so; eight warps a row with 128 registers 1.4 to 2 times as
  // long as now.
  constexpr int U = 16 / RD;
  constexpr int UK = WPR == 1 && RD > 2 ? 4 : 8;
  extern __shared__ float qs[];  // WPR 1: [ATT_WARPS][d]; else [d] and the warps' partial results [WPR][ATT_RESULT(RD)]
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const long long gw = WPR == 1 ? (long long)blockIdx.x * ATT_WARPS + warp : (long long)blockIdx.x;
  if (gw >= (long long)T_tokens * nq) return;
  const int t = (int)(gw / nq), h = (int)(gw - (long long)t * nq);
  const int kvh = h / (nq / nkv);
  // rows of the caches: which head of a page, how many heads it has, and where a value row of it starts
  const int pg_heads = shared_keys ? 1 : nkv, pg_h = shared_keys ? 0 : kvh;
  const int v_row = shared_keys ? nkv * v_ld : dv, v_off = shared_keys ? kvh * v_ld : 0;
  const int s = token_seq[t];
  const int qpos = positions[t];
  const int kend = qpos + 1;
  int kstart = (window > 0 && qpos - window + 1 > 0) ? qpos - window + 1 : 0;
  if (chunk > 0) kstart = max(kstart, qpos / chunk * chunk);
  // the kept first keys that lie ahead of the recent ones: a range of their own, walked first
  const int kept_end = (window > 0 && keep_first > 0) ? min(min(keep_first, kstart), kend) : 0;
  const int kept_start = (chunk > 0) ? min(qpos / chunk * chunk, kept_end) : 0;
  const float inv_cap = softcap > 0.f ? 1.0f / softcap : 0.f;
  const float slope = slopes ? slopes[h] : 0.f;
  float* myq = WPR == 1 ? qs + warp * d : qs;
  const T* qrow = q + (size_t)t * q_stride + (size_t)h * d;
  if (WPR == 1) {
    for (int i = lane; i < d; i += 32) myq[i] = to_f32(qrow[i]);
    __syncwarp();
  } else {
    for (int i = threadIdx.x; i < d; i += 32 * WPR) myq[i] = to_f32(qrow[i]);
    __syncthreads();
  }
  const int* bt = block_table + (size_t)s * max_blocks;

  // the row's parts, the kept range's and then the recent range's
  const int kept_first = kept_start / ATT_PART, kept_parts = kept_end > kept_start ? (kept_end - 1) / ATT_PART - kept_first + 1 : 0;
  const int first = kstart / ATT_PART, parts = kept_parts + (kend - 1) / ATT_PART - first + 1;
  float m_row = -INFINITY, l_row = 0.f, row[RD];
#pragma unroll
  for (int r = 0; r < RD; ++r) row[r] = 0.f;
  for (int p0 = 0; p0 < parts; p0 += WPR) {
    const int part = p0 + (WPR == 1 ? 0 : warp);
    float m = -INFINITY, l = 0.f, acc[RD];
    bool lost = false;               // a group whose scores are all NaN stood before the part's first score
#pragma unroll
    for (int r = 0; r < RD; ++r) acc[r] = 0.f;
    if (part < parts) {
      const bool kept = part < kept_parts;
      const int base = (kept ? kept_first + part : first + part - kept_parts) * ATT_PART;
      const int lo = max(kept ? kept_start : kstart, base), hi = min(kept ? kept_end : kend, base + ATT_PART);
      for (int j0 = (lo / 32) * 32; j0 < hi; j0 += 32) {
        const int j = j0 + lane;
        const bool valid = (j >= lo) && (j < hi);
        float score = -INFINITY;
        int page = -1;
        if (valid) {
          page = bt[j / page_size];
          if (page < 0 || page >= num_pages) {
            atomicOr(err, 4);
            page = -1;
          } else {
            const T* kp = kcache + (((size_t)page * pg_heads + pg_h) * page_size + (j % page_size)) * d;
            float dot = 0.f;
            if (VEC) {
#pragma unroll UK
              for (int i = 0; i < d; i += 8) {
                float kv[8];
                Vec8<T>::load(kp + i, kv);
#pragma unroll
                for (int u = 0; u < 8; ++u) dot = fmaf(myq[i + u], kv[u], dot);
              }
            } else {
#pragma unroll UK
              for (int i = 0; i < d; ++i) dot = fmaf(myq[i], to_f32(kp[i]), dot);
            }
            score = dot * scale;
            if (softcap > 0.f) score = softcap * tanhf(score * inv_cap);
            if (slopes) score -= slope * (float)(qpos - j);
          }
        }
        const float cmax = warp_max(score);
        const float m_new = fmaxf(m, cmax);
        if (m_new == -INFINITY) {          // nothing visible in this group (warp-uniform), or nothing but NaN
          lost |= __any_sync(0xffffffffu, score != score);
          continue;
        }
        const float p = (score == -INFINITY) ? 0.f : expf(score - m_new);
        const float corr = (m == -INFINITY) ? 0.f : expf(m - m_new);
        l = l * corr + warp_sum(p);
#pragma unroll
        for (int r = 0; r < RD; ++r) acc[r] *= corr;
        m = m_new;
        const int jn = min(32, hi - j0);
        for (int j8 = max(0, lo - j0) & ~(U - 1); j8 < jn; j8 += U) {
          float pj[U], v[U][RD];
#pragma unroll
          for (int u = 0; u < U; ++u) {
            pj[u] = __shfl_sync(0xffffffffu, p, j8 + u);
            const int pg = __shfl_sync(0xffffffffu, page, j8 + u);
            const T* vp = vcache + (((size_t)max(pg, 0) * pg_heads + pg_h) * page_size + ((j0 + j8 + u) % page_size)) * v_row + v_off;
#pragma unroll
            for (int r = 0; r < RD; ++r) v[u][r] = (pg >= 0 && lane + 32 * r < dv) ? to_f32(vp[lane + 32 * r]) : 0.f;
          }
#pragma unroll
          for (int u = 0; u < U; ++u)
#pragma unroll
            for (int r = 0; r < RD; ++r) acc[r] = fmaf(pj[u], v[u][r], acc[r]);       // a key that is not there: 0 * 0
        }
      }
    }
    // the partial results in order
    auto add = [&](float pm, float pl, const float (&pa)[RD], bool nan) {
      if (nan && m_row != -INFINITY) {            // as where the part's groups follow the row's others: the row is NaN
        l_row = NAN;
#pragma unroll
        for (int r = 0; r < RD; ++r) row[r] = NAN;
      }
      if (pm == -INFINITY) return;
      const float m_new = fmaxf(m_row, pm);
      const float old = (m_row == -INFINITY) ? 0.f : expf(m_row - m_new), now = expf(pm - m_new);
      l_row = l_row * old + pl * now;
#pragma unroll
      for (int r = 0; r < RD; ++r) row[r] = row[r] * old + pa[r] * now;
      m_row = m_new;
    };
    if (WPR == 1) {
      add(m, l, acc, lost);
    } else {
      float* mine = qs + d + warp * ATT_RESULT(RD);
#pragma unroll
      for (int r = 0; r < RD; ++r) mine[lane + 32 * r] = acc[r];
      if (lane == 0) { mine[32 * RD] = m; mine[32 * RD + 1] = l; mine[32 * RD + 2] = lost ? 1.f : 0.f; }
      __syncthreads();
      if (warp == 0)
        for (int w = 0; w < WPR && p0 + w < parts; ++w) {
          const float* theirs = qs + d + w * ATT_RESULT(RD);
#pragma unroll
          for (int r = 0; r < RD; ++r) acc[r] = theirs[lane + 32 * r];
          add(theirs[32 * RD], theirs[32 * RD + 1], acc, theirs[32 * RD + 2] != 0.f);
        }
      __syncthreads();
    }
  }
  if (WPR != 1 && warp != 0) return;
  if (sinks) {                                   // one more term of the denominator
    const float sk = sinks[h];
    const float m_new = fmaxf(m_row, sk);
    const float corr = (m_row == -INFINITY) ? 0.f : expf(m_row - m_new);
    l_row = l_row * corr + expf(sk - m_new);
#pragma unroll
    for (int r = 0; r < RD; ++r) row[r] *= corr;
  }
  T* orow = out + ((size_t)t * nq + h) * dv;
  float inv = (l_row > 0.f) ? 1.0f / l_row : 0.f;
  const T* grow = gate_mode ? gate + (size_t)t * gate_stride : nullptr;
  if (gate_mode == 1) inv *= 1.0f / (1.0f + expf(-to_f32(grow[h])));
#pragma unroll
  for (int r = 0; r < RD; ++r) {
    const int i = lane + 32 * r;
    if (i < dv) {
      float v = row[r] * inv;
      if (gate_mode == 2) v *= 1.0f / (1.0f + expf(-to_f32(grow[(size_t)h * dv + i])));
      orow[i] = from_f32<T>(v);
    }
  }
}

// keys [pages, nkv, page_size, d], values [pages, nkv, page_size, dv], out [T, nq * dv]; with shared_keys: keys
// [pages, 1, page_size, d], values [pages, 1, page_size, nkv * v_ld]
// How many warps share a row, of 1 and 8: eight where rows are few for the keys that they see.  The block table's width bounds
// the keys, and so do a window (with its kept keys) and a chunk; how long each sequence is, only the device knows (a wide
// table means a long row, which takes far longer with one warp than all short ones with eight).  Eight warps' time over
// one's, mean over float32 and bfloat16 heads of 64, 128 and 256: 512 rows x 128 keys 0.86, x 200 0.61; 1,024 x 200 1.03, x 256
// 0.88; 2,048 x 400 0.98, x 512 0.85; 4,096 x 512 0.95, x 800 0.79 and x 128 2.3.
RLLM_EXPORT int rllm_attention_simt_warps(long long rows, int max_blocks, int page_size, int window, int keep_first, int chunk) {
  long long keys = (long long)max_blocks * page_size;
  if (window > 0 && (long long)window + keep_first < keys) keys = (long long)window + keep_first;
  if (chunk > 0 && chunk < keys) keys = chunk;
  const long long enough = rows / 4 < 640 ? rows / 4 : 640;
  return rows <= 4096 && keys > ATT_PART && keys >= enough ? 8 : 1;
}

RLLM_EXPORT int rllm_attention_simt_kv(const void* q, int q_stride, void* out, const void* kcache,
                                       const void* vcache, int dtype, const int* block_table,
                                       int max_blocks, const int* positions, const int* token_seq, int T,
                                       int nq, int nkv, int d, int dv, int page_size, int num_pages, int window,
                                       float scale, int keep_first, int chunk, float softcap, const float* sinks,
                                       const void* gate, int gate_stride, int gate_mode, const float* slopes,
                                       int shared_keys, int v_ld, int* err, cudaStream_t stream) {
  if (T <= 0) return 0;
  if (nq <= 0 || nkv <= 0 || nq % nkv != 0 || d <= 0 || dv <= 0 || page_size <= 0 || num_pages <= 0 ||
      max_blocks <= 0 || window < 0 || keep_first < 0 || chunk < 0 || !(softcap >= 0.f) || gate_mode < 0 ||
      gate_mode > 2 || (gate_mode && !gate) || (shared_keys && v_ld < dv))
    return RLLM_E_BADARG;
  if (dv > ATT_MAX_D || d > 2816) return RLLM_E_UNSUPPORTED;
  const bool vec = d % 8 == 0 && q_stride % 8 == 0 && (((uintptr_t)q | (uintptr_t)kcache) & 31) == 0;
  const long long rows = (long long)T * nq;
  const bool share = rllm_attention_simt_warps(rows, max_blocks, page_size, window, keep_first, chunk) == 8;
  const unsigned blocks = (unsigned)(share ? rows : (rows + ATT_WARPS - 1) / ATT_WARPS);
  const int rd = dv <= 64 ? 2 : (dv <= 128 ? 4 : 8);
  const size_t smem = (share ? (size_t)d + 8 * ATT_RESULT(rd) : (size_t)ATT_WARPS * d) * sizeof(float);
#define ATT_ONE(VEC_, RD_, WPR_)                                                                            \
  RLLM_DISPATCH_DTYPE(dtype, T_,                                                                            \
    (attention_simt_kernel<T_, VEC_, RD_, WPR_><<<blocks, 32 * (WPR_ == 1 ? ATT_WARPS : WPR_), smem, stream>>>(  \
        (const T_*)q, q_stride, (T_*)out, (const T_*)kcache, (const T_*)vcache, block_table,                \
        max_blocks, positions, token_seq, T, nq, nkv, d, dv, page_size, num_pages, window, scale, keep_first,  \
        chunk, softcap, sinks, (const T_*)gate, gate_stride, gate_mode, slopes, shared_keys, v_ld, err)))
#define ATT_GO(VEC_)                                                                                        \
  do {                                                                                                      \
    if (share) { if (rd == 2) ATT_ONE(VEC_, 2, 8); else if (rd == 4) ATT_ONE(VEC_, 4, 8); else ATT_ONE(VEC_, 8, 8); }  \
    else { if (rd == 2) ATT_ONE(VEC_, 2, 1); else if (rd == 4) ATT_ONE(VEC_, 4, 1); else ATT_ONE(VEC_, 8, 1); }        \
  } while (0)
  if (vec) ATT_GO(true); else ATT_GO(false);
#undef ATT_ONE
#undef ATT_GO
  RLLM_LAUNCH_CHECK();
  return 0;
}

RLLM_EXPORT int rllm_attention_simt(const void* q, int q_stride, void* out, const void* kcache,
                                    const void* vcache, int dtype, const int* block_table,
                                    int max_blocks, const int* positions, const int* token_seq, int T,
                                    int nq, int nkv, int d, int page_size, int num_pages, int window,
                                    float scale, int* err, cudaStream_t stream) {
  if (d % 16 != 0 || d > ATT_MAX_D) return d > 0 ? RLLM_E_UNSUPPORTED : RLLM_E_BADARG;  // head sizes in steps of 16, to 256
  if (q_stride % 8 != 0) return RLLM_E_BADARG;
  return rllm_attention_simt_kv(q, q_stride, out, kcache, vcache, dtype, block_table, max_blocks, positions,
                                token_seq, T, nq, nkv, d, d, page_size, num_pages, window, scale, 0, 0, 0.f, nullptr,
                                nullptr, 0, 0, nullptr, 0, 0, err, stream);
}
