// Causal softmax attention over the paged cache, for any mix of new tokens: whole
// prompts, pieces of prompts, or one token per sequence.  One block per (token, head).
// This is the general kernel: it serves the float32 path and every shape; the
// bfloat16 path uses the specialised kernels in attention_prefill.cu and
// attention_decode.cu where they apply.
//
// Reference: for query head h the key/value head is h / (n_heads / n_kv_heads);
// s_i = (q . K[t_i]) * scale over the causal range only, p = softmax(s) with the
// maximum subtracted, out = sum_i p_i V[t_i]   (src/transformer/gqa_scalar.c:61-121,
// prefill: src/transformer/batched_attn_scalar.c:97-169).  The online form with a
// running maximum and sum is the reference's flash variant (gqa_scalar.c:127-207).
#include "common.cuh"

#define ATT_THREADS 128
#define ATT_CHUNK 128

template <typename T>
struct Vec16;
template <>
struct Vec16<float> {
  static constexpr int N = 4;
  __device__ static void load(const float* p, float* o) {
    float4 v = *reinterpret_cast<const float4*>(p);
    o[0] = v.x; o[1] = v.y; o[2] = v.z; o[3] = v.w;
  }
};
template <>
struct Vec16<__nv_bfloat16> {
  static constexpr int N = 8;
  __device__ static void load(const __nv_bfloat16* p, float* o) {
    uint4 v = *reinterpret_cast<const uint4*>(p);
    const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&v);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      float2 f = __bfloat1622float2(h[i]);
      o[2 * i] = f.x; o[2 * i + 1] = f.y;
    }
  }
};

// 1 / (l + e^(sink - m)) for sums l taken relative to the maximum m, also when the sink exceeds every score
__device__ __forceinline__ float sink_inverse(float m, float l, float sink) {
  const float top = fmaxf(m, sink);
  const float a = expf(m - top);
  return a / (l * a + expf(sink - top));
}

// a result number: in the compute type, or (out_wide) as float32 into an output that is a float32 array
template <typename T>
__device__ __forceinline__ void store_result(T* out, int out_wide, size_t at, float v) {
  if (out_wide) reinterpret_cast<float*>(out)[at] = v;
  else out[at] = from_f32<T>(v);
}

// Optional extras, each off when its pointer is null or its number zero, so that one kernel
// serves every softmax attention of the library:
//   v_dim        width of a value head when it differs from a key head's
//   keep_first   with a window: keys at positions below keep_first stay visible however far back
//   rel, n_rel   additive bias by distance, rel[min(pos - p, n_rel - 1) * n_heads + h] (float32; the
//                scale does not multiply it)
//   gate         per token and head a number whose logistic function multiplies the head's output
//   out_scale    a factor on all of the output (1: none)
//   chunk        positions are cut into chunks of this many and a token sees the earlier keys of its own
//                chunk only (takes the place of the window)
//   v_row        width of a row of the value plane when it is more than v_dim: the values are the first
//                v_dim numbers of each row (the key plane itself, for values that are a part of the keys)
//   sink         per head a score (float32) that stands in the softmax's denominator once, without a key and
//                without a value: the weights then sum to less than one
//   out_wide     the output is a float32 array whatever the compute type (what follows wants the sums unrounded)
//   v_share      so many consecutive key heads read one value head (the value plane has n_kv_heads / v_share
//                heads): several maps of scores over the same values
template <typename T>
__global__ void attention_general_kernel(const T* __restrict__ q, int q_stride, T* __restrict__ out,
                                         int out_stride, int n_heads, int n_kv_heads, int head_dim, int v_dim,
                                         float scale, int window, int keep_first, int chunk, int v_row,
                                         const float* __restrict__ rel, int n_rel, const T* __restrict__ gate, int gate_stride,
                                         const int* __restrict__ tok_seq,
                                         const int* __restrict__ tok_pos, const int* __restrict__ slots,
                                         const int* __restrict__ page_table, int pt_stride,
                                         const T* __restrict__ k_cache, const T* __restrict__ v_cache,
                                         float* __restrict__ part, int n_splits, const float* __restrict__ sink, int v_share, int out_wide, float out_scale) {
  pdl_launch_dependents();  // the next kernel in the stream may begin its prologue
  pdl_wait();               // the kernels before this one have completed and their writes are visible
  extern __shared__ __align__(16) float sm[];
  float* qs = sm;                    // head_dim
  float* ps = qs + head_dim;         // ATT_CHUNK scores, then probabilities
  float* scratch = ps + ATT_CHUNK;   // 32
  int t = blockIdx.x, h = blockIdx.y;
  int kvh = h / (n_heads / n_kv_heads);
  const int vh = kvh / v_share, n_v_heads = n_kv_heads / v_share;
  int pos = tok_pos[t];
  const int* pt = page_table + (size_t)slots[tok_seq[t]] * pt_stride;
  int lo = chunk > 0 ? (pos / chunk) * chunk : (window > 0 ? max(0, pos - window + 1) : 0);
  // visible keys: positions [0, n_first) and [lo, pos]; u counts through both ranges
  int n_first = min(keep_first, lo);
  int n_keys = n_first + pos - lo + 1;

  const T* qrow = q + (size_t)t * q_stride + (size_t)h * head_dim;
  for (int d = threadIdx.x; d < head_dim; d += blockDim.x) qs[d] = to_f32<T>(qrow[d]);
  __syncthreads();

  constexpr int VN = Vec16<T>::N;
  constexpr int MAX_D = 8;  // output dims per thread when a row is not read in 16-byte pieces: v_dim <= 1024
  // Weighted sum of the values.  Rows of whole 16-byte pieces: a row is read by v_dim / VN threads,
  // one piece each, and the rows of a chunk are shared out over the groups of such threads; the
  // groups' sums meet in shared memory at the end.  Other widths: one thread per dimension.
  const bool wide = (v_dim % VN) == 0 && (v_row % VN) == 0 && v_dim / VN <= ATT_THREADS;
  const int per_row = wide ? v_dim / VN : 1, groups = wide ? ATT_THREADS / per_row : 1;
  const int piece = threadIdx.x % per_row, group = threadIdx.x / per_row;
  float acc[MAX_D];
#pragma unroll
  for (int r = 0; r < MAX_D; ++r) acc[r] = 0.f;
  float accv[VN];
#pragma unroll
  for (int e = 0; e < VN; ++e) accv[e] = 0.f;
  float m_run = -INFINITY, l_run = 0.f;

  // with n_splits > 1 the chunks of keys are dealt out to the blocks blockIdx.z = 0 .. n_splits - 1, which
  // leave their running maximum, sum and unnormalised output in `part` for attention_merge_kernel
  for (int base = blockIdx.z * ATT_CHUNK; base < n_keys; base += ATT_CHUNK * n_splits) {
    int n = min(ATT_CHUNK, n_keys - base);
    float s = -INFINITY;
    if ((int)threadIdx.x < n) {
      int u = base + threadIdx.x;
      int p = u < n_first ? u : lo + (u - n_first);
      const T* krow = k_cache + cache_row_offset(pt, p, n_kv_heads, kvh, head_dim);
      float dot = 0.f;
      if (head_dim % VN == 0) {  // rows of whole 16-byte pieces
        for (int d = 0; d < head_dim; d += VN) {
          float kv[VN];
          Vec16<T>::load(krow + d, kv);
          const float4* q4 = reinterpret_cast<const float4*>(qs + d);  // four numbers of q per read
#pragma unroll
          for (int e = 0; e < VN / 4; ++e) {
            const float4 a = q4[e];
            dot = fmaf(a.x, kv[4 * e], dot); dot = fmaf(a.y, kv[4 * e + 1], dot);
            dot = fmaf(a.z, kv[4 * e + 2], dot); dot = fmaf(a.w, kv[4 * e + 3], dot);
          }
        }
      } else {
        for (int d = 0; d < head_dim; ++d) dot = fmaf(qs[d], to_f32<T>(krow[d]), dot);
      }
      s = dot * scale;
      if (rel) s += rel[(size_t)min(pos - p, n_rel - 1) * n_heads + h];
    }
    float m_chunk = block_max(s, scratch);
    float m_new = fmaxf(m_run, m_chunk);
    float alpha = (m_run == -INFINITY) ? 0.f : expf(m_run - m_new);
    float p_mine = ((int)threadIdx.x < n) ? expf(s - m_new) : 0.f;
    ps[threadIdx.x] = p_mine;
    float l_chunk = block_sum(p_mine, scratch);  // has the barrier that publishes ps[]
    l_run = l_run * alpha + l_chunk;
    m_run = m_new;
    if (wide) {
#pragma unroll
      for (int e = 0; e < VN; ++e) accv[e] *= alpha;
      if (group < groups) {
        for (int j = group; j < n; j += groups) {
          int u = base + j;
          int p = u < n_first ? u : lo + (u - n_first);
          float vv[VN];
          Vec16<T>::load(v_cache + cache_row_offset(pt, p, n_v_heads, vh, v_row) + piece * VN, vv);
          float w = ps[j];
#pragma unroll
          for (int e = 0; e < VN; ++e) accv[e] = fmaf(w, vv[e], accv[e]);
        }
      }
    } else {
#pragma unroll
      for (int r = 0; r < MAX_D; ++r) {
        int d = threadIdx.x + r * ATT_THREADS;
        if (d < v_dim) {
          float a = acc[r] * alpha;
          for (int j = 0; j < n; ++j) {
            int u = base + j;
            int p = u < n_first ? u : lo + (u - n_first);
            const T* vrow = v_cache + cache_row_offset(pt, p, n_v_heads, vh, v_row);
            a = fmaf(ps[j], to_f32<T>(vrow[d]), a);
          }
          acc[r] = a;
        }
      }
    }
    __syncthreads();  // ps[] is rewritten by the next chunk
  }
  float inv = sink && !part ? sink_inverse(m_run, l_run, sink[h]) : 1.0f / l_run;
  if (gate) inv *= 1.0f / (1.0f + expf(-to_f32<T>(gate[(size_t)t * gate_stride + h])));
  inv *= out_scale;
  const size_t orow = (size_t)t * out_stride + (size_t)h * v_dim;
  float* prow = part ? part + (((size_t)t * n_heads + h) * n_splits + blockIdx.z) * (v_dim + 2) : nullptr;
  if (prow && threadIdx.x == 0) { prow[0] = m_run; prow[1] = l_run; }
  if (wide) {
    // groups * v_dim <= ATT_THREADS * VN floats, kept behind the scores
    float* red = scratch + 32;
    if (group < groups) {
#pragma unroll
      for (int e = 0; e < VN; ++e) red[(size_t)group * v_dim + piece * VN + e] = accv[e];
    }
    __syncthreads();
    for (int d = threadIdx.x; d < v_dim; d += ATT_THREADS) {
      float a = 0.f;
      for (int g = 0; g < groups; ++g) a += red[(size_t)g * v_dim + d];
      if (prow) prow[2 + d] = a;
      else store_result<T>(out, out_wide, orow + d, a * inv);
    }
    return;
  }
#pragma unroll
  for (int r = 0; r < MAX_D; ++r) {
    int d = threadIdx.x + r * ATT_THREADS;
    if (d < v_dim) {
      if (prow) prow[2 + d] = acc[r];
      else store_result<T>(out, out_wide, orow + d, acc[r] * inv);
    }
  }
}

// The same for R query heads of one key/value head at once (a block per token and group of R heads): every key
// and value row is read once for the R heads instead of once per head, which is what bounds the kernel above when
// many heads share few rows (one token per sequence, grouped or multi-query heads: the rows come from the L2 R
// times less often).  Rows of whole 16-byte pieces only (head_dim, v_dim, v_row multiples of the piece).
template <int R>
__device__ __forceinline__ void block_max_sum_r(float* v, float* scratch, bool is_max) {
  // v[R] per thread -> the block's maximum (or sum) of each, to every thread; scratch holds 32 * R floats
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarp = (blockDim.x + 31) >> 5;
#pragma unroll
  for (int r = 0; r < R; ++r) v[r] = is_max ? warp_max(v[r]) : warp_sum(v[r]);
  __syncthreads();
  if (lane == 0) {
#pragma unroll
    for (int r = 0; r < R; ++r) scratch[warp * R + r] = v[r];
  }
  __syncthreads();
#pragma unroll
  for (int r = 0; r < R; ++r) {
    float a = is_max ? -INFINITY : 0.f;
    for (int w = 0; w < nwarp; ++w) a = is_max ? fmaxf(a, scratch[w * R + r]) : a + scratch[w * R + r];
    v[r] = a;
  }
}

template <typename T, int R>
__global__ void __launch_bounds__(ATT_THREADS)
attention_grouped_kernel(const T* __restrict__ q, int q_stride, T* __restrict__ out, int out_stride, int n_heads,
                         int n_kv_heads, int head_dim, int v_dim, float scale, int window, int keep_first, int chunk,
                         int v_row, const float* __restrict__ rel, int n_rel, const T* __restrict__ gate, int gate_stride,
                         const int* __restrict__ tok_seq, const int* __restrict__ tok_pos, const int* __restrict__ slots,
                         const int* __restrict__ page_table, int pt_stride, const T* __restrict__ k_cache,
                         const T* __restrict__ v_cache, float* __restrict__ part, int n_splits,
                         const float* __restrict__ sink, int v_share, int out_wide, float out_scale) {
  pdl_launch_dependents();
  pdl_wait();
  extern __shared__ __align__(16) float sm[];
  float* qs = sm;                           // [R][head_dim]
  float* ps = qs + (size_t)R * head_dim;    // [R][ATT_CHUNK] probabilities
  float* scratch = ps + R * ATT_CHUNK;      // [32 * R]
  float* red = scratch + 32 * R;            // [R][groups * v_dim] at the end
  const int t = blockIdx.x, h0 = blockIdx.y * R;
  const int kvh = h0 / (n_heads / n_kv_heads);
  const int vh = kvh / v_share, n_v_heads = n_kv_heads / v_share;
  const int pos = tok_pos[t];
  const int* pt = page_table + (size_t)slots[tok_seq[t]] * pt_stride;
  const int lo = chunk > 0 ? (pos / chunk) * chunk : (window > 0 ? max(0, pos - window + 1) : 0);
  const int n_first = min(keep_first, lo);
  const int n_keys = n_first + pos - lo + 1;
  constexpr int VN = Vec16<T>::N;
  for (int i = threadIdx.x; i < R * head_dim; i += blockDim.x)
    qs[i] = to_f32<T>(q[(size_t)t * q_stride + (size_t)h0 * head_dim + i]);
  __syncthreads();
  const int per_row = v_dim / VN, groups = ATT_THREADS / per_row;
  const int piece = threadIdx.x % per_row, group = threadIdx.x / per_row;
  float accv[R][VN];
#pragma unroll
  for (int r = 0; r < R; ++r)
#pragma unroll
    for (int e = 0; e < VN; ++e) accv[r][e] = 0.f;
  float m_run[R], l_run[R];
#pragma unroll
  for (int r = 0; r < R; ++r) { m_run[r] = -INFINITY; l_run[r] = 0.f; }

  for (int base = blockIdx.z * ATT_CHUNK; base < n_keys; base += ATT_CHUNK * n_splits) {
    const int n = min(ATT_CHUNK, n_keys - base);
    float s[R];
#pragma unroll
    for (int r = 0; r < R; ++r) s[r] = -INFINITY;
    if ((int)threadIdx.x < n) {
      const int u = base + threadIdx.x;
      const int p = u < n_first ? u : lo + (u - n_first);
      const T* krow = k_cache + cache_row_offset(pt, p, n_kv_heads, kvh, head_dim);
      float dot[R];
#pragma unroll
      for (int r = 0; r < R; ++r) dot[r] = 0.f;
#pragma unroll 8
      for (int d = 0; d < head_dim; d += VN) {
        float kv[VN];
        Vec16<T>::load(krow + d, kv);
#pragma unroll
        for (int r = 0; r < R; ++r) {
          const float4* q4 = reinterpret_cast<const float4*>(qs + r * head_dim + d);  // four numbers of q per read
#pragma unroll
          for (int e = 0; e < VN / 4; ++e) {
            const float4 a = q4[e];
            dot[r] = fmaf(a.x, kv[4 * e], dot[r]); dot[r] = fmaf(a.y, kv[4 * e + 1], dot[r]);
            dot[r] = fmaf(a.z, kv[4 * e + 2], dot[r]); dot[r] = fmaf(a.w, kv[4 * e + 3], dot[r]);
          }
        }
      }
#pragma unroll
      for (int r = 0; r < R; ++r) {
        s[r] = dot[r] * scale;
        if (rel) s[r] += rel[(size_t)min(pos - p, n_rel - 1) * n_heads + h0 + r];
      }
    }
    float m_new[R], alpha[R], p_mine[R];
#pragma unroll
    for (int r = 0; r < R; ++r) m_new[r] = s[r];
    block_max_sum_r<R>(m_new, scratch, true);
#pragma unroll
    for (int r = 0; r < R; ++r) {
      m_new[r] = fmaxf(m_run[r], m_new[r]);
      alpha[r] = (m_run[r] == -INFINITY) ? 0.f : expf(m_run[r] - m_new[r]);
      p_mine[r] = ((int)threadIdx.x < n) ? expf(s[r] - m_new[r]) : 0.f;
      ps[r * ATT_CHUNK + threadIdx.x] = p_mine[r];
    }
    block_max_sum_r<R>(p_mine, scratch, false);  // has the barriers that publish ps[]
#pragma unroll
    for (int r = 0; r < R; ++r) {
      l_run[r] = l_run[r] * alpha[r] + p_mine[r];
      m_run[r] = m_new[r];
#pragma unroll
      for (int e = 0; e < VN; ++e) accv[r][e] *= alpha[r];
    }
    if (group < groups) {
      // eight rows of values in flight at a time: a row alone leaves the thread waiting for its one load
      constexpr int VB = 8;
      for (int j0 = group; j0 < n; j0 += VB * groups) {
        float vv[VB][VN];
#pragma unroll
        for (int b = 0; b < VB; ++b) {
          const int j = j0 + b * groups;
          if (j < n) {
            const int u = base + j;
            const int p = u < n_first ? u : lo + (u - n_first);
            Vec16<T>::load(v_cache + cache_row_offset(pt, p, n_v_heads, vh, v_row) + piece * VN, vv[b]);
          }
        }
#pragma unroll
        for (int b = 0; b < VB; ++b) {
          const int j = j0 + b * groups;
          if (j < n) {
#pragma unroll
            for (int r = 0; r < R; ++r) {
              const float w = ps[r * ATT_CHUNK + j];
#pragma unroll
              for (int e = 0; e < VN; ++e) accv[r][e] = fmaf(w, vv[b][e], accv[r][e]);
            }
          }
        }
      }
    }
    __syncthreads();  // ps[] is rewritten by the next chunk
  }
  // the groups' sums meet in shared memory: red[r][group][v_dim]
  if (group < groups) {
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
      for (int e = 0; e < VN; ++e) red[((size_t)r * groups + group) * v_dim + piece * VN + e] = accv[r][e];
  }
  __syncthreads();
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const int h = h0 + r;
    float inv = sink && !part ? sink_inverse(m_run[r], l_run[r], sink[h]) : 1.0f / l_run[r];
    if (gate) inv *= 1.0f / (1.0f + expf(-to_f32<T>(gate[(size_t)t * gate_stride + h])));
    inv *= out_scale;
    const size_t orow = (size_t)t * out_stride + (size_t)h * v_dim;
    float* prow = part ? part + (((size_t)t * n_heads + h) * n_splits + blockIdx.z) * (v_dim + 2) : nullptr;
    if (prow && threadIdx.x == 0) { prow[0] = m_run[r]; prow[1] = l_run[r]; }
    for (int d = threadIdx.x; d < v_dim; d += ATT_THREADS) {
      float a = 0.f;
      for (int g = 0; g < groups; ++g) a += red[((size_t)r * groups + g) * v_dim + d];
      if (prow) prow[2 + d] = a;
      else store_result<T>(out, out_wide, orow + d, a * inv);
    }
  }
}

// out[t][h] = sum_z e^{m_z - M} acc_z / sum_z e^{m_z - M} l_z (times the logistic function of the gate), M = max_z m_z
template <typename T>
__global__ void attention_merge_kernel(const float* __restrict__ part, int n_splits, int n_heads, int v_dim,
                                       const T* __restrict__ gate, int gate_stride, T* __restrict__ out, int out_stride,
                                       const float* __restrict__ sink, int out_wide, float out_scale) {
  pdl_launch_dependents();
  pdl_wait();
  // Bound by latency: the parts' maxima and sums are one load per lane, their weights are worked out once, and a thread's numbers
  // are asked for eight at a time.
  __shared__ float weight[64];  // at most 64 splits
  __shared__ float s_inv;
  const int t = blockIdx.x, h = blockIdx.y;
  const float* p = part + ((size_t)t * n_heads + h) * n_splits * (v_dim + 2);
  if (threadIdx.x < 32) {
    float m[2], l[2], M = -INFINITY, L = 0.f;
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int z = threadIdx.x + 32 * i;
      m[i] = z < n_splits ? p[(size_t)z * (v_dim + 2)] : -INFINITY;
      l[i] = z < n_splits ? p[(size_t)z * (v_dim + 2) + 1] : 0.f;
      M = fmaxf(M, m[i]);
    }
    M = warp_max(M);
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const float w = m[i] != -INFINITY ? expf(m[i] - M) : -1.f;  // (a part without keys holds nothing and is passed over)
      if (m[i] != -INFINITY) L += w * l[i];
      weight[threadIdx.x + 32 * i] = w;
    }
    L = warp_sum(L);
    if (threadIdx.x == 0) {
      float inv = sink ? sink_inverse(M, L, sink[h]) : 1.0f / L;
      if (gate) inv *= 1.0f / (1.0f + expf(-to_f32<T>(gate[(size_t)t * gate_stride + h])));
      s_inv = inv * out_scale;
    }
  }
  __syncthreads();
  const float inv = s_inv;
  for (int d = threadIdx.x; d < v_dim; d += blockDim.x) {
    float a = 0.f;
    for (int z0 = 0; z0 < n_splits; z0 += 8) {
      float v[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) v[i] = z0 + i < n_splits ? p[(size_t)(z0 + i) * (v_dim + 2) + 2 + d] : 0.f;
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const float w = z0 + i < n_splits ? weight[z0 + i] : -1.f;
        if (!(w < 0.f)) a = fmaf(w, v[i], a);  // also with a weight of zero: times not a number it is none
      }
    }
    store_result<T>(out, out_wide, (size_t)t * out_stride + (size_t)h * v_dim + d, a * inv);
  }
}

// ---- few tokens in bfloat16 on the tensor cores ---------------------------------------------------
// A block takes one token, up to 16 query heads of one key/value head and, of every n_splits x 64 visible keys, 64.  Their key and
// value rows are copied into shared memory (two stages where both fit), every row once for all the heads; four warps take 16 keys
// each for the scores (mma.sync m16n8k16, heads as the 16 rows; the inner dimension is taken in the order in which 16-byte pieces
// lie in a lane, the same for both operands) and a quarter of the value width each for the weighted sum.  The weights enter that
// product as three bfloat16 terms, 24 bits of mantissa, so nothing is rounded that float32 would not round; values inside the key
// rows are read from the same copy.
// Scores are summed over 32 numbers of the inner dimension and weighted rows over 16 keys on the tensor cores, from zero each time; the
// rest is float32 additions.  The tensor cores cut their sums off where an addition rounds: left in their accumulators, the results
// were 1.2 (16 keys) to 18 times (4,000) as far from 64 bits as sums in float32, now 0.3 to 1.04 times, for 3 to 8 % of the time.
// Bound by latency: a token's keys are few kilobytes per block.  The kernel above spends 4,300 instructions per warp on 128 keys
// of 128 numbers, this one some 300.  Measured with the merge, us, that kernel and this (tokens, heads, key/value heads, head size, visible keys):
// 4, 16, 4, 128, 1024: 16.0 / 10.6;  1, 32, 8, 128, 4000: 25.6 / 16.6;  64, 32, 8, 128, 2000: 534 / 297;  key rows of 256 that hold values
// of 192, 8, 16, 1, 1000: 31.9 / 13.4;  of 576 and 512, 2, 32, 1, 1024: 42.6 / 25.8.
#define AM_THREADS 128
#define AM_KEYS 64
#define AM_P_PITCH 144  // bytes of 64 weights, padded: no bank conflicts between rows
struct AmArgs {
  const __nv_bfloat16* q;
  int q_stride;
  void* out;
  int out_stride, n_heads, n_kv_heads, head_dim, v_dim;
  float scale;
  int window, keep_first, chunk, v_row;
  const float* rel;
  int n_rel;
  const __nv_bfloat16* gate;
  int gate_stride;
  const int *tok_seq, *tok_pos, *slots, *page_table;
  int pt_stride;
  const __nv_bfloat16 *k_cache, *v_cache;
  float* part;
  int n_splits;
  const float* sink;
  int v_share, out_wide;
  float out_scale;
  int tiles_per_group;  // blocks of 16 heads per key/value head
  int shared_rows;      // the values are a part of the key rows
  int stages;
  int q_pitch, k_pitch, v_pitch;  // bytes of a row in shared memory
};
__device__ __forceinline__ void am_copy(unsigned dst, const __nv_bfloat16* src, bool live) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(live ? 16 : 0) : "memory");
}
__device__ __forceinline__ uint4 am_piece(unsigned addr) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr) : "memory");
  return v;
}
__device__ __forceinline__ void am_mma(float* c, unsigned a0, unsigned a1, unsigned a2, unsigned a3, unsigned b0, unsigned b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

template <int NT>  // tiles of 8 value dimensions per warp
__global__ void __launch_bounds__(AM_THREADS) attention_few_mma_kernel(AmArgs a) {
  pdl_launch_dependents();
  pdl_wait();
  extern __shared__ __align__(16) unsigned char am_smem[];
  __shared__ int s_row[2][AM_KEYS];         // page x 64 + row of a stage's keys, -1: none
  __shared__ float s_m[4][16], s_l[4][16];  // per warp and head
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, quad = lane & 3;
  const int t = blockIdx.x, kvh = blockIdx.y / a.tiles_per_group, z = blockIdx.z;
  const int gq = a.n_heads / a.n_kv_heads, first_head = (blockIdx.y % a.tiles_per_group) * 16;
  const int h0 = kvh * gq + first_head, rows = min(16, gq - first_head);
  const int vh = kvh / a.v_share, n_v_heads = a.n_kv_heads / a.v_share;
  const int pos = a.tok_pos[t];
  const int* pt = a.page_table + (size_t)a.slots[a.tok_seq[t]] * a.pt_stride;
  const int lo = a.chunk > 0 ? (pos / a.chunk) * a.chunk : (a.window > 0 ? max(0, pos - a.window + 1) : 0);
  const int n_first = min(a.keep_first, lo), n_keys = n_first + pos - lo + 1;
  const int pieces = a.head_dim / 8, q_pieces = (a.head_dim + 31) / 32 * 4, v_pieces = a.v_dim / 8;

  const unsigned base = (unsigned)__cvta_generic_to_shared(am_smem);
  const unsigned qs = base, ps = qs + 16 * a.q_pitch, ks0 = ps + 3 * 16 * AM_P_PITCH;
  const unsigned stage_bytes = AM_KEYS * (a.k_pitch + a.v_pitch);  // v_pitch 0: values in the key rows
  auto position = [&](int u) { return u < n_first ? u : lo + (u - n_first); };
  auto fill = [&](int it) {
    const int u0 = (it * a.n_splits + z) * AM_KEYS, st = it % a.stages;
    if (tid < AM_KEYS) {
      const int u = u0 + tid, p = position(u);
      s_row[st][tid] = u < n_keys ? pt[p / BN_PAGE] * BN_PAGE + p % BN_PAGE : -1;
    }
    __syncthreads();
    const unsigned kd = ks0 + st * stage_bytes, vd = kd + AM_KEYS * a.k_pitch;
    for (int i = tid; i < AM_KEYS * q_pieces; i += AM_THREADS) {  // (pieces past the head size are zeros)
      const int r = i / q_pieces, c = i - r * q_pieces, at = s_row[st][r];
      const bool live = at >= 0 && c < pieces;
      am_copy(kd + r * a.k_pitch + c * 16,
              live ? a.k_cache + (((size_t)(at / BN_PAGE) * a.n_kv_heads + kvh) * BN_PAGE + at % BN_PAGE) * a.head_dim + c * 8 : a.k_cache, live);
    }
    if (!a.shared_rows)
      for (int i = tid; i < AM_KEYS * v_pieces; i += AM_THREADS) {
        const int r = i / v_pieces, c = i - r * v_pieces, at = s_row[st][r];
        am_copy(vd + r * a.v_pitch + c * 16,
                at >= 0 ? a.v_cache + (((size_t)(at / BN_PAGE) * n_v_heads + vh) * BN_PAGE + at % BN_PAGE) * a.v_row + c * 8 : a.v_cache, at >= 0);
      }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  const int span = a.n_splits * AM_KEYS;
  const int turns = n_keys > z * AM_KEYS ? (n_keys - z * AM_KEYS + span - 1) / span : 0;
  if (turns > 0) {  // a part without keys copies nothing: what it leaves does not depend on q, and nothing would wait for the copy
    for (int i = tid; i < 16 * q_pieces; i += AM_THREADS) {
      const int r = i / q_pieces, c = i - r * q_pieces;
      const bool live = r < rows && c < pieces;
      am_copy(qs + r * a.q_pitch + c * 16, live ? a.q + (size_t)t * a.q_stride + (size_t)(h0 + r) * a.head_dim + c * 8 : a.q, live);
    }
    fill(0);  // (q's copy is in the first stage's group)
  }

  float o[NT][4];
#pragma unroll
  for (int j = 0; j < NT; ++j)
#pragma unroll
    for (int e = 0; e < 4; ++e) o[j][e] = 0.f;
  float m_run[2] = {-INFINITY, -INFINITY}, l_run[2] = {0.f, 0.f};  // heads g and g + 8; the sums of this lane's keys
  for (int it = 0; it < turns; ++it) {
    if (a.stages == 2 && it + 1 < turns) {
      fill(it + 1);
      asm volatile("cp.async.wait_group 1;" ::: "memory");
    } else {
      asm volatile("cp.async.wait_group 0;" ::: "memory");
    }
    __syncthreads();
    const int u0 = (it * a.n_splits + z) * AM_KEYS, st = it % a.stages;
    const unsigned kd = ks0 + st * stage_bytes;
    const unsigned vd = a.shared_rows ? kd : kd + AM_KEYS * a.k_pitch, v_pitch = a.shared_rows ? a.k_pitch : a.v_pitch;
    // scores of this warp's 16 keys
    float s[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
    const unsigned xa = qs + g * a.q_pitch + quad * 16, ka = kd + (warp * 16 + g) * a.k_pitch + quad * 16;
#pragma unroll 4
    for (int c = 0; c < q_pieces; c += 4) {
      const uint4 x0 = am_piece(xa + c * 16);
      const uint4 x1 = rows > 8 ? am_piece(xa + 8 * a.q_pitch + c * 16) : make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
      for (int n = 0; n < 2; ++n) {
        const uint4 k = am_piece(ka + n * 8 * a.k_pitch + c * 16);
        float d[4] = {0.f, 0.f, 0.f, 0.f};
        am_mma(d, x0.x, x1.x, x0.y, x1.y, k.x, k.y);
        am_mma(d, x0.z, x1.z, x0.w, x1.w, k.z, k.w);
#pragma unroll
        for (int e = 0; e < 4; ++e) s[n][e] += d[e];
      }
    }
    float mx[2] = {-INFINITY, -INFINITY};
#pragma unroll
    for (int n = 0; n < 2; ++n)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int u = u0 + warp * 16 + n * 8 + quad * 2 + (e & 1), head = g + (e >> 1) * 8;
        float v = -INFINITY;
        if (u < n_keys) {
          v = s[n][e] * a.scale;
          if (a.rel && head < rows) v += a.rel[(size_t)min(pos - position(u), a.n_rel - 1) * a.n_heads + h0 + head];
        }
        s[n][e] = v;
        mx[e >> 1] = fmaxf(mx[e >> 1], v);
      }
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      mx[i] = fmaxf(mx[i], __shfl_xor_sync(0xffffffffu, mx[i], 1));
      mx[i] = fmaxf(mx[i], __shfl_xor_sync(0xffffffffu, mx[i], 2));
      if (quad == 0) s_m[warp][g + 8 * i] = mx[i];
    }
    __syncthreads();
    float alpha[2];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      float m = m_run[i];
#pragma unroll
      for (int w = 0; w < 4; ++w) m = fmaxf(m, s_m[w][g + 8 * i]);
      alpha[i] = m_run[i] == -INFINITY ? 0.f : expf(m_run[i] - m);
      m_run[i] = m;
      l_run[i] *= alpha[i];
    }
#pragma unroll
    for (int j = 0; j < NT; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e) o[j][e] *= alpha[e >> 1];
    // the weights, as three bfloat16 terms each
#pragma unroll
    for (int n = 0; n < 2; ++n)
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        float w0 = s[n][2 * i] == -INFINITY ? 0.f : expf(s[n][2 * i] - m_run[i]);
        float w1 = s[n][2 * i + 1] == -INFINITY ? 0.f : expf(s[n][2 * i + 1] - m_run[i]);
        l_run[i] += w0 + w1;
        const unsigned dst = ps + (g + 8 * i) * AM_P_PITCH + (warp * 16 + n * 8 + quad * 2) * 2;
#pragma unroll
        for (int term = 0; term < 3; ++term) {
          const __nv_bfloat162 both = __floats2bfloat162_rn(w0, w1);
          asm volatile("st.shared.u32 [%0], %1;" ::"r"(dst + term * 16 * AM_P_PITCH), "r"(*reinterpret_cast<const unsigned*>(&both)) : "memory");
          w0 -= __low2float(both);
          w1 -= __high2float(both);
        }
      }
    __syncthreads();
    // this warp's share of the value dimensions
#pragma unroll
    for (int kk = 0; kk < AM_KEYS / 16; ++kk) {
      unsigned p[3][4];
#pragma unroll
      for (int term = 0; term < 3; ++term)
        asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
                     : "=r"(p[term][0]), "=r"(p[term][1]), "=r"(p[term][2]), "=r"(p[term][3])
                     : "r"(ps + (term * 16 + (lane & 15)) * AM_P_PITCH + (kk * 16 + (lane >> 4) * 8) * 2) : "memory");
#pragma unroll
      for (int j = 0; j < NT; ++j) {
        const int tile = warp * NT + j;
        if (tile >= v_pieces) continue;  // the same for the whole warp
        unsigned b0, b1;
        asm volatile("ldmatrix.sync.aligned.m8n8.x2.trans.shared.b16 {%0, %1}, [%2];"
                     : "=r"(b0), "=r"(b1) : "r"(vd + (kk * 16 + (lane & 15)) * v_pitch + tile * 16) : "memory");
        float d[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int term = 2; term >= 0; --term) am_mma(d, p[term][0], p[term][1], p[term][2], p[term][3], b0, b1);  // the small ones first
#pragma unroll
        for (int e = 0; e < 4; ++e) o[j][e] += d[e];
      }
    }
    __syncthreads();  // keys, values and weights have been used
    if (a.stages == 1 && it + 1 < turns) fill(it + 1);
  }
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    l_run[i] += __shfl_xor_sync(0xffffffffu, l_run[i], 1);
    l_run[i] += __shfl_xor_sync(0xffffffffu, l_run[i], 2);
    if (quad == 0) s_l[warp][g + 8 * i] = l_run[i];
    if (quad == 0 && warp == 0) s_m[0][g + 8 * i] = m_run[i];  // (the same for every warp)
  }
  float zero = 0.f;  // not a number where a sum is not finite
#pragma unroll
  for (int j = 0; j < NT; ++j)
#pragma unroll
    for (int e = 0; e < 4; ++e) zero = fmaf(0.f, o[j][e], zero);
  const bool all_finite = !__syncthreads_or(zero != 0.f);  // (the last turn has waited for every copy)
  auto sum_of = [&](int head) { return (s_l[0][head] + s_l[1][head]) + (s_l[2][head] + s_l[3][head]); };
  auto factor = [&](int head, float m, float l) {
    const int h = h0 + head;
    float inv = a.sink ? sink_inverse(m, l, a.sink[h]) : 1.0f / l;
    if (a.gate) inv *= 1.0f / (1.0f + expf(-__bfloat162float(a.gate[(size_t)t * a.gate_stride + h])));
    return inv * a.out_scale;
  };
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const int head = g + 8 * i;
    if (head >= rows) continue;
    const int h = h0 + head;
    const float l = sum_of(head);
    if (a.part) {
      float* prow = a.part + (((size_t)t * a.n_heads + h) * a.n_splits + z) * (a.v_dim + 2);
      if (warp == 0 && quad == 0) { prow[0] = m_run[i]; prow[1] = l; }
#pragma unroll
      for (int j = 0; j < NT; ++j) {
        const int d = (warp * NT + j) * 8 + quad * 2;
        if (d < a.v_dim) { prow[2 + d] = o[j][2 * i]; prow[3 + d] = o[j][2 * i + 1]; }
      }
    } else {
      const float inv = factor(head, m_run[i], l);
      const size_t orow = (size_t)t * a.out_stride + (size_t)h * a.v_dim;
#pragma unroll
      for (int j = 0; j < NT; ++j) {
        const int d = (warp * NT + j) * 8 + quad * 2;
        if (d < a.v_dim) {
          store_result<__nv_bfloat16>((__nv_bfloat16*)a.out, a.out_wide, orow + d, o[j][2 * i] * inv);
          store_result<__nv_bfloat16>((__nv_bfloat16*)a.out, a.out_wide, orow + d + 1, o[j][2 * i + 1] * inv);
        }
      }
    }
  }
  if (all_finite) return;
  // A value of infinity times the lower terms of its weight, which may be zero or of the other sign, made a sum that is not a number,
  // where one in float32 is infinite.  Looked for only in sums that are not finite; a value or a weight that is not a number, and
  // infinities of both signs, leave them as they are.
  __syncthreads();  // the block's results have been written
  for (int i = tid; i < rows * a.v_dim; i += AM_THREADS) {
    const int head = i / a.v_dim, d = i - head * a.v_dim;
    float* p = a.part ? a.part + (((size_t)t * a.n_heads + h0 + head) * a.n_splits + z) * (a.v_dim + 2) + 2 + d : nullptr;
    const size_t at = (size_t)t * a.out_stride + (size_t)(h0 + head) * a.v_dim + d;
    const float is = p ? *p : load_as_f32(a.out, a.out_wide ? BN_F32 : BN_BF16, at), l = sum_of(head);
    bool up = false, down = false, none = l != l;
    if (fabsf(is) < INFINITY || none) continue;
    for (int u0 = z * AM_KEYS; u0 < n_keys; u0 += span)
      for (int u = u0; u < min(u0 + AM_KEYS, n_keys); ++u) {
        const int pos_u = position(u);
        const float v = __bfloat162float(
            a.v_cache[(((size_t)pt[pos_u / BN_PAGE] * n_v_heads + vh) * BN_PAGE + pos_u % BN_PAGE) * a.v_row + d]);
        up |= v == INFINITY;
        down |= v == -INFINITY;
        none |= v != v;
      }
    if (none || up == down) continue;
    const float o = up ? INFINITY : -INFINITY;
    if (p) *p = o;
    else store_result<__nv_bfloat16>((__nv_bfloat16*)a.out, a.out_wide, at, o * factor(head, s_m[0][head], l));
  }
}

#define AM_MAX_V_DIM 512
#define AM_SMEM_MAX (200 * 1024)
// Shared memory of the kernel above; fills in pitches and stages.
static size_t am_layout(AmArgs* a) {
  const int q_bytes = (a->head_dim + 31) / 32 * 64;
  a->q_pitch = q_bytes % 128 ? q_bytes : q_bytes + 64;  // eight lanes read two rows' pieces without a conflict
  a->k_pitch = a->shared_rows ? (q_bytes + 127) / 128 * 128 + 16 : a->q_pitch;  // ldmatrix reads eight rows
  a->v_pitch = a->shared_rows ? 0 : (a->v_dim * 2 + 127) / 128 * 128 + 16;
  const size_t fixed = (size_t)16 * a->q_pitch + 3 * 16 * AM_P_PITCH, stage = (size_t)AM_KEYS * (a->k_pitch + a->v_pitch);
  a->stages = fixed + 2 * stage <= 112 * 1024 ? 2 : 1;
  return fixed + a->stages * stage;
}
// Whether the kernel above is built for these sizes: whole 16-byte pieces, value rows and shared memory that fit.
extern "C" int bn_attention_few_fits(int head_dim, int v_dim, int v_row, int q_stride, int shared_rows) {
  AmArgs a = {};
  a.head_dim = head_dim; a.v_dim = v_dim; a.shared_rows = shared_rows;
  return head_dim > 0 && v_dim > 0 && head_dim % 8 == 0 && v_dim % 8 == 0 && v_row % 8 == 0 && q_stride % 8 == 0 && v_dim <= AM_MAX_V_DIM &&
         am_layout(&a) <= AM_SMEM_MAX;
}
template <int NT>
static int am_launch(const AmArgs& a, dim3 grid, size_t smem, cudaStream_t stream) {
  static BnGrant grant;
  cudaError_t e = grant.ask((const void*)attention_few_mma_kernel<NT>, smem, 2048);
  if (e != cudaSuccess) return BN_ERR_LAUNCH + (int)e;
  BN_LAUNCH(attention_few_mma_kernel<NT>, grid, AM_THREADS, smem, stream, a);
  return BN_OK;
}

// q: [n_tokens, q_stride] with head h at element h*head_dim; out [n_tokens, out_stride] with head h at
// element h*v_dim.  The keys and values of the new tokens must already be in the cache.  few: on the tensor cores, a block per token
// (bfloat16 of sizes that bn_attention_few_fits, q and the caches 16-byte aligned; n_splits then deals out 64 keys at a time).
extern "C" int bn_attention_general_ex(const void* q, int q_stride, void* out, int out_stride, int dtype,
                                       int n_tokens, int n_heads, int n_kv_heads, int head_dim, int v_dim, float scale,
                                       int window, int keep_first, int chunk, int v_row, const float* rel, int n_rel,
                                       const void* gate, int gate_stride, const int* tok_seq, const int* tok_pos, const int* slots,
                                       const int* page_table, int pt_stride,
                                       const void* k_cache, const void* v_cache, float* part, int n_splits,
                                       const float* sink, int v_share, int out_wide, float out_scale, int few, cudaStream_t stream) {
  if (n_tokens <= 0) return BN_OK;
  if (v_share < 1 || n_kv_heads % v_share || (v_share > 1 && v_row > 0)) return BN_ERR_BAD_ARG;
  if (n_splits < 1 || n_splits > 64 || (n_splits > 1 && !part)) return BN_ERR_BAD_ARG;
  if (n_splits == 1) part = nullptr;
  if (v_row <= 0) v_row = v_dim;
  // value rows of whole 16-byte pieces may be up to 128 pieces wide; others are one dimension per thread, eight times
  const int vn = dtype == BN_F32 ? 4 : 8;
  const bool wide = v_dim % vn == 0 && v_row % vn == 0 && v_dim / vn <= ATT_THREADS;
  if (head_dim <= 0 || head_dim > 2048 || n_kv_heads <= 0 || n_heads % n_kv_heads || window < 0 || keep_first < 0 ||
      chunk < 0 || (chunk > 0 && (window > 0 || keep_first > 0)) || v_dim <= 0 || v_row < v_dim ||
      (!wide && v_dim > 8 * ATT_THREADS) || (rel && n_rel <= 0))
    return BN_ERR_BAD_ARG;
  if (n_heads > 65535) return BN_ERR_BAD_ARG;
  if (few) {
    AmArgs am = {};
    am.q = (const __nv_bfloat16*)q; am.q_stride = q_stride; am.out = out; am.out_stride = out_stride; am.n_heads = n_heads;
    am.n_kv_heads = n_kv_heads; am.head_dim = head_dim; am.v_dim = v_dim; am.scale = scale; am.window = window; am.keep_first = keep_first;
    am.chunk = chunk; am.v_row = v_row; am.rel = rel; am.n_rel = n_rel; am.gate = (const __nv_bfloat16*)gate; am.gate_stride = gate_stride;
    am.tok_seq = tok_seq; am.tok_pos = tok_pos; am.slots = slots; am.page_table = page_table; am.pt_stride = pt_stride;
    am.k_cache = (const __nv_bfloat16*)k_cache; am.v_cache = (const __nv_bfloat16*)v_cache; am.part = part; am.n_splits = n_splits;
    am.sink = sink; am.v_share = v_share; am.out_wide = out_wide; am.out_scale = out_scale;
    am.tiles_per_group = (n_heads / n_kv_heads + 15) / 16;
    am.shared_rows = v_cache == k_cache && v_row == head_dim && v_share == 1 && v_dim <= head_dim;
    if (dtype != BN_BF16 || !bn_attention_few_fits(head_dim, v_dim, v_row, q_stride, am.shared_rows) ||
        (((uintptr_t)q | (uintptr_t)k_cache | (uintptr_t)v_cache) & 15))
      return BN_ERR_BAD_ARG;
    const size_t smem = am_layout(&am);
    const dim3 agrid(n_tokens, n_kv_heads * am.tiles_per_group, n_splits);
    const int rc = v_dim <= 32 ? am_launch<1>(am, agrid, smem, stream) : v_dim <= 64 ? am_launch<2>(am, agrid, smem, stream) :
                   v_dim <= 128 ? am_launch<4>(am, agrid, smem, stream) : v_dim <= 256 ? am_launch<8>(am, agrid, smem, stream) :
                   am_launch<16>(am, agrid, smem, stream);
    if (rc != BN_OK) return rc;
    if (part)
      BN_LAUNCH((attention_merge_kernel<__nv_bfloat16>), dim3(n_tokens, n_heads), 128, 0, stream, (const float*)part, n_splits, n_heads, v_dim,
                (const __nv_bfloat16*)gate, gate_stride, (__nv_bfloat16*)out, out_stride, sink, out_wide, out_scale);
    BN_CHECK_LAUNCH();
    return BN_OK;
  }
  // few tokens whose heads share rows: the heads of a key/value head four (or two) at a time, rows read once for them
  const int gq = n_heads / n_kv_heads;
  const int R = (gq % 4 == 0) ? 4 : ((gq % 2 == 0) ? 2 : 1);
  if (R > 1 && wide && head_dim % vn == 0 && n_tokens <= 256) {
    dim3 ggrid(n_tokens, n_heads / R, n_splits);
    const size_t gsmem = ((size_t)R * head_dim + R * ATT_CHUNK + 32 * R + (size_t)R * ATT_THREADS * vn) * sizeof(float);
#define BN_GROUPED(TT, RR)                                                                                                  \
  do {                                                                                                                      \
    if (gsmem > 48 * 1024) {                                                                                                \
      static size_t granted = 0;                                                                                            \
      if (gsmem > granted) {                                                                                                \
        cudaError_t e = cudaFuncSetAttribute(attention_grouped_kernel<TT, RR>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)gsmem); \
        if (e != cudaSuccess) return BN_ERR_LAUNCH + (int)e;                                                                \
        granted = gsmem;                                                                                                    \
      }                                                                                                                     \
    }                                                                                                                       \
    BN_LAUNCH((attention_grouped_kernel<TT, RR>), ggrid, ATT_THREADS, gsmem, stream, (const TT*)q, q_stride, (TT*)out,       \
              out_stride, n_heads, n_kv_heads, head_dim, v_dim, scale, window, keep_first, chunk, v_row, rel, n_rel,        \
              (const TT*)gate, gate_stride, tok_seq, tok_pos, slots, page_table, pt_stride, (const TT*)k_cache,              \
              (const TT*)v_cache, part, n_splits, sink, v_share, out_wide, out_scale);                                                           \
  } while (0)
    if (gsmem <= 160 * 1024 && (dtype == BN_F32 || dtype == BN_BF16)) {
      if (dtype == BN_F32) { if (R == 4) BN_GROUPED(float, 4); else BN_GROUPED(float, 2); }
      else { if (R == 4) BN_GROUPED(__nv_bfloat16, 4); else BN_GROUPED(__nv_bfloat16, 2); }
#undef BN_GROUPED
      if (part) {
        dim3 mgrid(n_tokens, n_heads);
        if (dtype == BN_F32)
          BN_LAUNCH((attention_merge_kernel<float>), mgrid, 128, 0, stream, (const float*)part, n_splits, n_heads, v_dim,
                    (const float*)gate, gate_stride, (float*)out, out_stride, sink, out_wide, out_scale);
        else
          BN_LAUNCH((attention_merge_kernel<__nv_bfloat16>), mgrid, 128, 0, stream, (const float*)part, n_splits, n_heads, v_dim,
                    (const __nv_bfloat16*)gate, gate_stride, (__nv_bfloat16*)out, out_stride, sink, out_wide, out_scale);
      }
      BN_CHECK_LAUNCH();
      return BN_OK;
    }
  }
  dim3 grid(n_tokens, n_heads, n_splits);
  size_t smem = (head_dim + ATT_CHUNK + 32 + ATT_THREADS * 8) * sizeof(float);  // q, scores, reduction scratch, the groups' sums
  if (dtype == BN_F32)
    BN_LAUNCH((attention_general_kernel<float>), grid, ATT_THREADS, smem, stream, 
        (const float*)q, q_stride, (float*)out, out_stride, n_heads, n_kv_heads, head_dim, v_dim, scale, window,
        keep_first, chunk, v_row, rel, n_rel, (const float*)gate, gate_stride,
        tok_seq, tok_pos, slots, page_table, pt_stride, (const float*)k_cache, (const float*)v_cache, part, n_splits, sink, v_share, out_wide, out_scale);
  else if (dtype == BN_BF16)
    BN_LAUNCH((attention_general_kernel<__nv_bfloat16>), grid, ATT_THREADS, smem, stream, 
        (const __nv_bfloat16*)q, q_stride, (__nv_bfloat16*)out, out_stride, n_heads, n_kv_heads, head_dim, v_dim,
        scale, window, keep_first, chunk, v_row, rel, n_rel, (const __nv_bfloat16*)gate, gate_stride,
        tok_seq, tok_pos, slots, page_table, pt_stride,
        (const __nv_bfloat16*)k_cache, (const __nv_bfloat16*)v_cache, part, n_splits, sink, v_share, out_wide, out_scale);
  else
    return BN_ERR_BAD_ARG;
  if (part) {
    dim3 mgrid(n_tokens, n_heads);
    if (dtype == BN_F32)
      BN_LAUNCH((attention_merge_kernel<float>), mgrid, 128, 0, stream, (const float*)part, n_splits, n_heads, v_dim,
                (const float*)gate, gate_stride, (float*)out, out_stride, sink, out_wide, out_scale);
    else
      BN_LAUNCH((attention_merge_kernel<__nv_bfloat16>), mgrid, 128, 0, stream, (const float*)part, n_splits, n_heads, v_dim,
                (const __nv_bfloat16*)gate, gate_stride, (__nv_bfloat16*)out, out_stride, sink, out_wide, out_scale);
  }
  BN_CHECK_LAUNCH();
  return BN_OK;
}

extern "C" int bn_attention_general(const void* q, int q_stride, void* out, int out_stride, int dtype,
                                    int n_tokens, int n_heads, int n_kv_heads, int head_dim, float scale,
                                    int window, const int* tok_seq, const int* tok_pos, const int* slots,
                                    const int* page_table, int pt_stride,
                                    const void* k_cache, const void* v_cache, cudaStream_t stream) {
  return bn_attention_general_ex(q, q_stride, out, out_stride, dtype, n_tokens, n_heads, n_kv_heads, head_dim, head_dim,
                                 scale, window, 0, 0, 0, nullptr, 0, nullptr, 0, tok_seq, tok_pos, slots, page_table,
                                 pt_stride, k_cache, v_cache, nullptr, 1, nullptr, 1, 0, 1.0f, 0, stream);
}
