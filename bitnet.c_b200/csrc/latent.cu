// Keys and values per head from cached latents, for runs of new tokens (bfloat16): the rows [latent | rotated key part] that a
// step's tokens see are read back from the pages, two products make every head's unrotated keys and values of the latents,
// and these go, with the shared rotated part behind each head's keys, into scratch pages that the attention kernels for runs
// of tokens read as if they were the cache.
//
//   bn_latent_gather  the latents of the seen positions, side by side: [seen, rank]
//   bn_latent_pages   keys [pages, heads, 64, dim + rot], values [pages, heads, 64, vdim]
//
// And the two products per head around attention in the latent space, for the few tokens of a decode step:
//
//   bn_latent_queries  ql[t, h] = [W_uk[h]^T q[t, h, :dim] | q[t, h, dim:]]
//   bn_latent_values   o[t, h] = W_uv[h] out[t, h]
//
// They are a few hundred kilobytes of weights each and bound by latency.  As the library's batched products (with a copy for the rotated
// parts) they took 2.8 + 2.4 and 2.9 us, and since those kernels neither begin before their predecessor has ended nor let their
// successor do so, attention took 11 instead of 8 us and the output product 10 instead of 5: per layer some 12 us more than here.
// A block has its share of a head's weights in registers before its input is there, and goes through the tokens with them.
#include "common.cuh"

// The cache row of seen position i
__device__ __forceinline__ const __nv_bfloat16* latent_row(const __nv_bfloat16* cache, int row, const int* seen_seq, const int* seen_pos,
                                                           const int* slots, const int* page_table, int pt_stride, int i) {
  const int p = seen_pos[i];
  return cache + ((size_t)page_table[(size_t)slots[seen_seq[i]] * pt_stride + p / BN_PAGE] * BN_PAGE + p % BN_PAGE) * row;
}

__global__ void latent_gather_kernel(const __nv_bfloat16* __restrict__ cache, int row, int rank, const int* __restrict__ seen_seq,
                                     const int* __restrict__ seen_pos, int n_seen, const int* __restrict__ slots,
                                     const int* __restrict__ page_table, int pt_stride, __nv_bfloat16* __restrict__ out) {
  pdl_launch_dependents();
  pdl_wait();
  const int i = blockIdx.x * blockDim.y + threadIdx.y;
  if (i >= n_seen) return;
  const __nv_bfloat16* src = latent_row(cache, row, seen_seq, seen_pos, slots, page_table, pt_stride, i);
  for (int c = threadIdx.x * 8; c < rank; c += blockDim.x * 8)
    *reinterpret_cast<uint4*>(out + (size_t)i * rank + c) = *reinterpret_cast<const uint4*>(src + c);
}

// A block per seen position; scratch_table [sequences, scratch_stride]: the scratch page of each page of a sequence.
__global__ void latent_pages_kernel(const __nv_bfloat16* __restrict__ keys, const __nv_bfloat16* __restrict__ values,
                                    const __nv_bfloat16* __restrict__ cache, int row, int rank, int heads, int dim, int rot, int vdim,
                                    const int* __restrict__ seen_seq, const int* __restrict__ seen_pos, const int* __restrict__ slots,
                                    const int* __restrict__ page_table, int pt_stride, const int* __restrict__ scratch_table,
                                    int scratch_stride, __nv_bfloat16* __restrict__ k_pages, __nv_bfloat16* __restrict__ v_pages) {
  pdl_launch_dependents();
  pdl_wait();
  const int i = blockIdx.x, pos = seen_pos[i];
  const __nv_bfloat16* turned = latent_row(cache, row, seen_seq, seen_pos, slots, page_table, pt_stride, i) + rank;
  const size_t page = scratch_table[(size_t)seen_seq[i] * scratch_stride + pos / BN_PAGE];
  const int r = pos % BN_PAGE, kd = dim + rot, per_key = kd / 8, per_value = vdim / 8;
  for (int j = threadIdx.x; j < heads * per_key; j += blockDim.x) {
    const int h = j / per_key, c = (j - h * per_key) * 8;
    const __nv_bfloat16* src = c < dim ? keys + ((size_t)i * heads + h) * dim + c : turned + c - dim;
    *reinterpret_cast<uint4*>(k_pages + ((page * heads + h) * BN_PAGE + r) * kd + c) = *reinterpret_cast<const uint4*>(src);
  }
  for (int j = threadIdx.x; j < heads * per_value; j += blockDim.x) {
    const int h = j / per_value, c = (j - h * per_value) * 8;
    *reinterpret_cast<uint4*>(v_pages + ((page * heads + h) * BN_PAGE + r) * vdim + c) =
        *reinterpret_cast<const uint4*>(values + ((size_t)i * heads + h) * vdim + c);
  }
}

// cache: pages of 64 rows of `row` bfloat16 numbers (one key head); seen_seq / seen_pos [n_seen]; out [n_seen, rank].  row and rank
// multiples of 8, 16-byte aligned.
extern "C" int bn_latent_gather(const void* cache, int row, int rank, const int* seen_seq, const int* seen_pos, int n_seen, const int* slots,
                                const int* page_table, int pt_stride, void* out, cudaStream_t stream) {
  if (n_seen <= 0) return BN_OK;
  if (!cache || !seen_seq || !seen_pos || !slots || !page_table || !out || rank <= 0 || rank > row || row % 8 || rank % 8 ||
      (((uintptr_t)cache | (uintptr_t)out) & 15))
    return BN_ERR_BAD_ARG;
  BN_LAUNCH(latent_gather_kernel, (n_seen + 3) / 4, dim3(64, 4), 0, stream, (const __nv_bfloat16*)cache, row, rank, seen_seq, seen_pos, n_seen,
            slots, page_table, pt_stride, (__nv_bfloat16*)out);
  return BN_OK;
}

// keys [n_seen, heads, dim], values [n_seen, heads, vdim]; k_pages [pages, heads, 64, row - rank + dim], v_pages [pages, heads, 64,
// vdim]; rows that no seen position fills are left alone.  All widths multiples of 8, all buffers 16-byte aligned.
extern "C" int bn_latent_pages(const void* keys, const void* values, const void* cache, int row, int rank, int heads, int dim, int vdim,
                               const int* seen_seq, const int* seen_pos, int n_seen, const int* slots, const int* page_table, int pt_stride,
                               const int* scratch_table, int scratch_stride, void* k_pages, void* v_pages, cudaStream_t stream) {
  if (n_seen <= 0) return BN_OK;
  if (!keys || !values || !cache || !seen_seq || !seen_pos || !slots || !page_table || !scratch_table || !k_pages || !v_pages || heads <= 0 ||
      dim <= 0 || vdim <= 0 || rank <= 0 || rank > row || row % 8 || rank % 8 || dim % 8 || vdim % 8 ||
      (((uintptr_t)keys | (uintptr_t)values | (uintptr_t)cache | (uintptr_t)k_pages | (uintptr_t)v_pages) & 15))
    return BN_ERR_BAD_ARG;
  BN_LAUNCH(latent_pages_kernel, n_seen, 256, 0, stream, (const __nv_bfloat16*)keys, (const __nv_bfloat16*)values, (const __nv_bfloat16*)cache, row,
            rank, heads, dim, row - rank, vdim, seen_seq, seen_pos, slots, page_table, pt_stride, scratch_table, scratch_stride,
            (__nv_bfloat16*)k_pages, (__nv_bfloat16*)v_pages);
  return BN_OK;
}

#define LT_THREADS 256
#define LT_DIM_MAX 256    // a thread holds 16 bytes of every 32nd row of W_uk[h]
#define LT_COLS 64        // columns of the latent space per block
#define LT_TOKENS 4       // tokens between two meetings of a block's warps
// grid (heads, ceil(rank / 64)).  Threads: 8 columns each of 64, and every 32nd number of the head; the parts meet within the warp, then in
// shared memory, in a fixed order.
__global__ void __launch_bounds__(LT_THREADS) latent_queries_kernel(const __nv_bfloat16* __restrict__ q, long long q_stride, int head_stride,
                                                                    const __nv_bfloat16* __restrict__ uk, int tokens, int dim, int rot, int rank,
                                                                    __nv_bfloat16* __restrict__ out) {
  pdl_launch_dependents();
  __shared__ __align__(16) float parts[LT_TOKENS][LT_THREADS / 32][LT_COLS];
  const int h = blockIdx.x, heads = gridDim.x, c0 = blockIdx.y * LT_COLS, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int cg = (tid & 7) * 8, d0 = tid >> 3;
  uint4 w[LT_DIM_MAX / 32];
#pragma unroll
  for (int i = 0; i < LT_DIM_MAX / 32; ++i) {
    w[i] = make_uint4(0u, 0u, 0u, 0u);
    const int d = d0 + 32 * i;
    if (d < dim && c0 + cg < rank) w[i] = *reinterpret_cast<const uint4*>(uk + ((size_t)h * dim + d) * rank + c0 + cg);
  }
  pdl_wait();
  const int row = rank + rot;
  for (int t0 = 0; t0 < tokens; t0 += LT_TOKENS) {
    float x[LT_TOKENS][LT_DIM_MAX / 32];
#pragma unroll
    for (int t = 0; t < LT_TOKENS; ++t)
#pragma unroll
      for (int i = 0; i < LT_DIM_MAX / 32; ++i) {
        const int d = d0 + 32 * i;
        x[t][i] = t0 + t < tokens && d < dim ? __bfloat162float(q[(t0 + t) * q_stride + (long long)h * head_stride + d]) : 0.f;
      }
#pragma unroll
    for (int t = 0; t < LT_TOKENS; ++t) {
      float s[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) s[j] = 0.f;
#pragma unroll
      for (int i = 0; i < LT_DIM_MAX / 32; ++i)
        if (32 * i < dim && t0 + t < tokens) {
          const unsigned u[4] = {w[i].x, w[i].y, w[i].z, w[i].w};
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            s[2 * j] = fmaf(x[t][i], __uint_as_float(u[j] << 16), s[2 * j]);
            s[2 * j + 1] = fmaf(x[t][i], __uint_as_float(u[j] & 0xffff0000u), s[2 * j + 1]);
          }
        }
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        s[j] += __shfl_xor_sync(0xffffffffu, s[j], 8);
        s[j] += __shfl_xor_sync(0xffffffffu, s[j], 16);
      }
      if (lane < 8) {
        *reinterpret_cast<float4*>(&parts[t][warp][cg]) = make_float4(s[0], s[1], s[2], s[3]);
        *reinterpret_cast<float4*>(&parts[t][warp][cg + 4]) = make_float4(s[4], s[5], s[6], s[7]);
      }
    }
    __syncthreads();
    {
      const int t = tid / LT_COLS, c = tid % LT_COLS;
      if (t0 + t < tokens && c0 + c < rank) {
        float v = 0.f;
#pragma unroll
        for (int i = 0; i < LT_THREADS / 32; ++i) v += parts[t][i][c];
        out[((size_t)(t0 + t) * heads + h) * row + c0 + c] = __float2bfloat16_rn(v);
      }
    }
    if (blockIdx.y == 0)
      for (int i = tid; i < LT_TOKENS * rot; i += LT_THREADS) {
        const int t = t0 + i / rot, j = i % rot;
        if (t < tokens) out[((size_t)t * heads + h) * row + rank + j] = q[t * q_stride + (long long)h * head_stride + dim + j];
      }
    __syncthreads();
  }
}

#define LT_ROWS 4          // rows of W_uv[h] per warp
#define LT_PIECES 2        // pieces of 256 numbers of the latent space (rank up to 512)
// grid (heads, ceil(vdim / 32)): a warp takes four rows, its lanes share out the latent space.
__global__ void __launch_bounds__(LT_THREADS) latent_values_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ uv,
                                                                   int tokens, int rank, int vdim, __nv_bfloat16* __restrict__ out) {
  pdl_launch_dependents();
  const int h = blockIdx.x, heads = gridDim.x, lane = threadIdx.x & 31;
  const int v0 = (blockIdx.y * (LT_THREADS / 32) + (threadIdx.x >> 5)) * LT_ROWS;
  float w[LT_ROWS][LT_PIECES][8];
#pragma unroll
  for (int r = 0; r < LT_ROWS; ++r)
#pragma unroll
    for (int p = 0; p < LT_PIECES; ++p) {
      const int c = p * 256 + lane * 8;
      uint4 v = make_uint4(0u, 0u, 0u, 0u);
      if (v0 + r < vdim && c < rank) v = *reinterpret_cast<const uint4*>(uv + ((size_t)h * vdim + v0 + r) * rank + c);
      const unsigned u[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        w[r][p][2 * j] = __uint_as_float(u[j] << 16);
        w[r][p][2 * j + 1] = __uint_as_float(u[j] & 0xffff0000u);
      }
    }
  pdl_wait();
  if (v0 >= vdim) return;
#pragma unroll 2
  for (int t = 0; t < tokens; ++t) {
    float s[LT_ROWS];
#pragma unroll
    for (int r = 0; r < LT_ROWS; ++r) s[r] = 0.f;
#pragma unroll
    for (int p = 0; p < LT_PIECES; ++p) {
      const int c = p * 256 + lane * 8;
      if (c >= rank) continue;
      const uint4 v = *reinterpret_cast<const uint4*>(x + ((size_t)t * heads + h) * rank + c);
      const unsigned u[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float lo = __uint_as_float(u[j] << 16), hi = __uint_as_float(u[j] & 0xffff0000u);
#pragma unroll
        for (int r = 0; r < LT_ROWS; ++r) s[r] = fmaf(hi, w[r][p][2 * j + 1], fmaf(lo, w[r][p][2 * j], s[r]));
      }
    }
    __syncwarp();
#pragma unroll
    for (int r = 0; r < LT_ROWS; ++r) s[r] = warp_sum(s[r]);
    const float mine = lane == 0 ? s[0] : lane == 1 ? s[1] : lane == 2 ? s[2] : s[3];
    if (lane < LT_ROWS && v0 + lane < vdim) out[((size_t)t * heads + h) * vdim + v0 + lane] = __float2bfloat16_rn(mine);
  }
}

// q: rows q_stride apart, of head h the numbers from h * head_stride on: dim unrotated ones and rot rotated; uk [heads, dim, rank]; out
// [tokens, heads, rank + rot].  rank a multiple of 8, dim up to 256, uk 16-byte aligned.
extern "C" int bn_latent_queries(const void* q, long long q_stride, int head_stride, const void* uk, int tokens, int heads, int dim, int rot,
                                 int rank, void* out, cudaStream_t stream) {
  if (tokens <= 0 || heads <= 0) return BN_OK;
  if (!q || !uk || !out || dim <= 0 || dim > LT_DIM_MAX || rot < 0 || rank <= 0 || rank % 8 || (rank + LT_COLS - 1) / LT_COLS > 65535 ||
      (uintptr_t)uk & 15)
    return BN_ERR_BAD_ARG;
  BN_LAUNCH(latent_queries_kernel, dim3(heads, (rank + LT_COLS - 1) / LT_COLS), LT_THREADS, 0, stream, (const __nv_bfloat16*)q, q_stride,
            head_stride, (const __nv_bfloat16*)uk, tokens, dim, rot, rank, (__nv_bfloat16*)out);
  return BN_OK;
}

// x [tokens, heads, rank], uv [heads, vdim, rank], out [tokens, heads, vdim].  rank a multiple of 8 up to 512; x and uv 16-byte aligned.
extern "C" int bn_latent_values(const void* x, const void* uv, int tokens, int heads, int rank, int vdim, void* out, cudaStream_t stream) {
  if (tokens <= 0 || heads <= 0) return BN_OK;
  const int per_block = LT_THREADS / 32 * LT_ROWS;
  if (!x || !uv || !out || rank <= 0 || rank % 8 || rank > 256 * LT_PIECES || vdim <= 0 || (vdim + per_block - 1) / per_block > 65535 ||
      ((uintptr_t)x | (uintptr_t)uv) & 15)
    return BN_ERR_BAD_ARG;
  BN_LAUNCH(latent_values_kernel, dim3(heads, (vdim + per_block - 1) / per_block), LT_THREADS, 0, stream, (const __nv_bfloat16*)x,
            (const __nv_bfloat16*)uv, tokens, rank, vdim, (__nv_bfloat16*)out);
  return BN_OK;
}
