// out[M, N] = x[M, K] . W[N, K]^T for few rows M: the weight matrix is streamed once per group
// of up to 8 rows of x.  Weights are row-major
// [out_features, in_features], y = W x, as in the reference (src/quant/f32_scalar.c:10-31);
// its decode path uses a warp-per-row matvec as well (src/gpu_cuda.cu:3976-4012).
// Products are accumulated in float32 whatever the storage type.
//
// float32 (linear_stream_f32_kernel): bound by the weights' bytes.  A block keeps its part of the rows of x (2,048 elements of
// each) in shared memory for as long as it runs; its warps each take a run of output columns, up to four at a time, and copy the
// weights' pieces asynchronously, every lane into slots of its own, several stages ahead and across the ends of columns.  A longer
// inner dimension is shared out over blockIdx.y in parts of 2,048, whose float32 sums a second small kernel adds in their
// order.  Measured, 8 rows, against a kernel that staged 1,024 elements of x at a time between barriers and held the weights in
// registers (us, before and after): 28672 x 4096 137 / 94 (5.0 TB/s), 4096 x 14336 72 / 54, 128256 x 4096 505 / 364 (5.8 TB/s),
// 6144 x 4096 38 / 34, 4096 x 4096 26 / 20; 16 rows of 28672 x 4096 263 / 180; one row 89 / 80.
//
// bfloat16 (linear_skinny_kernel; only matrices that the tensor-core kernels do not take): a block stages a chunk of the rows of x
// in shared memory; a warp takes two output columns and two 16-byte pieces of each per step, so that four weight loads are in
// flight per lane and what it reads of x serves both columns.
// A matrix with few rows has too few warps to keep the memory busy (4,096 rows are 256 blocks on 148
// SMs), so its inner dimension is shared out over blockIdx.y: split s takes the chunks s, s + splits,
// ... of x and leaves its float32 partial sums in a scratch buffer likewise.
//
// How many splits there are depends on the matrix alone (never on the rows of x),
// so the order of a result's additions does not depend on what else is in the batch.
#include "common.cuh"

template <typename T>
struct VecLd;
template <>
struct VecLd<__nv_bfloat16> {
  static constexpr int N = 8;
  __device__ static void unpack(uint4 v, float* o) {
    const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&v);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      float2 f = __bfloat1622float2(h[i]);
      o[2 * i] = f.x; o[2 * i + 1] = f.y;
    }
  }
  __device__ static void load(const __nv_bfloat16* p, float* o) { unpack(__ldg(reinterpret_cast<const uint4*>(p)), o); }
  __device__ static void load_shared(const __nv_bfloat16* p, float* o) { unpack(*reinterpret_cast<const uint4*>(p), o); }
};

#define SK_MT 8
#define SK_WARPS 8
#define SK_COLS 2   // output columns per warp
#define SK_KC 1024  // elements of a row of x staged at a time (SK_MT rows: 32 KB in float32)

template <typename T>
__global__ void __launch_bounds__(SK_WARPS * 32)
linear_skinny_kernel(const T* __restrict__ x, const T* __restrict__ w, void* __restrict__ out, int out_dtype, int M, int N,
                     int K, int ldo, float* __restrict__ partial, const float* __restrict__ bias) {
  pdl_launch_dependents();  // the next kernel in the stream may begin its prologue
  pdl_wait();               // the kernels before this one have completed and their writes are visible
  __shared__ __align__(16) T xs[SK_MT][SK_KC];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  constexpr int VN = VecLd<T>::N;
  const int n0 = (blockIdx.x * SK_WARPS + warp) * SK_COLS;
  const int nc = min(SK_COLS, N - n0);  // <= 0: this warp has no column, it only helps staging
  // columns past the matrix read the last one again (their sums are not stored)
  const T* wrow[SK_COLS];
#pragma unroll
  for (int c = 0; c < SK_COLS; ++c) wrow[c] = w + (size_t)min(n0 + c, N - 1) * K;
  for (int m0 = 0; m0 < M; m0 += SK_MT) {
    const int mt = min(SK_MT, M - m0);
    float acc[SK_MT][SK_COLS];
#pragma unroll
    for (int i = 0; i < SK_MT; ++i)
#pragma unroll
      for (int c = 0; c < SK_COLS; ++c) acc[i][c] = 0.f;
    for (int kc = blockIdx.y * SK_KC; kc < K; kc += gridDim.y * SK_KC) {
      const int kn = min(SK_KC, K - kc);  // a multiple of 8
      __syncthreads();  // the chunk before this one has been used by every warp
      for (int i = 0; i < mt; ++i)
        for (int kk = threadIdx.x * VN; kk < kn; kk += SK_WARPS * 32 * VN)
          *reinterpret_cast<uint4*>(&xs[i][kk]) = __ldg(reinterpret_cast<const uint4*>(x + (size_t)(m0 + i) * K + kc + kk));
      __syncthreads();
      if (nc <= 0) continue;
      // The order of the additions of one output depends on K alone: lane l adds the products of
      // elements l*VN.. of every piece of 32*VN elements in turn (two pieces per step), then the
      // lanes are summed by the same tree.
      for (int k = lane * VN; k < kn; k += 2 * 32 * VN) {
        const bool second = k + 32 * VN < kn;
        float wv[2][SK_COLS][VN];
#pragma unroll
        for (int c = 0; c < SK_COLS; ++c) {
          VecLd<T>::load(wrow[c] + kc + k, wv[0][c]);
          if (second) VecLd<T>::load(wrow[c] + kc + k + 32 * VN, wv[1][c]);
        }
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          if (u == 1 && !second) break;
#pragma unroll
          for (int i = 0; i < SK_MT; ++i) {
            if (i < mt) {
              float xv[VN];
              VecLd<T>::load_shared(&xs[i][k + u * 32 * VN], xv);
#pragma unroll
              for (int c = 0; c < SK_COLS; ++c)
#pragma unroll
                for (int e = 0; e < VN; ++e) acc[i][c] = fmaf(wv[u][c][e], xv[e], acc[i][c]);
            }
          }
        }
      }
    }
#pragma unroll
    for (int i = 0; i < SK_MT; ++i) {
      if (i < mt) {
#pragma unroll
        for (int c = 0; c < SK_COLS; ++c) {
          float v = warp_sum(acc[i][c]);
          if (lane == 0 && c < nc) {
            if (gridDim.y > 1) partial[((size_t)blockIdx.y * M + m0 + i) * N + n0 + c] = v;
            else store_from_f32(out, out_dtype, (size_t)(m0 + i) * ldo + n0 + c, bias ? v + bias[n0 + c] : v);
          }
        }
      }
    }
  }
}

// ---- float32 ----------------------------------------------------------------------------------
#define SF_THREADS 256
#define SF_WARPS (SF_THREADS / 32)
#define SF_KC 2048  // elements of the inner dimension per block
// Rows of x and ring together take 112 KB of shared memory, two blocks an SM's: the fewer rows, the longer the ring.  COLS: output
// columns a warp works on at a time; what it reads of x serves all of them, but a warp that has few must not leave their places
// in the ring empty.
__host__ __device__ constexpr int sf_stages(int MT, int COLS) { return (MT > 4 ? 12 : MT > 2 ? 20 : 24) / COLS; }
__host__ __device__ constexpr int sf_smem(int MT) { return MT * SF_KC * 4 + sf_stages(MT, 1) * 16 * SF_THREADS; }

// The sums over the warp's lanes of 32 numbers per lane, number l to lane l: the tree of warp_sum, each level for half as many
// numbers as the one before.
__device__ __forceinline__ float warp_sums_of_32(float* a, int lane) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
#pragma unroll
    for (int j = 0; j < o; ++j) {
      const float keep = (lane & o) ? a[j + o] : a[j], send = (lane & o) ? a[j] : a[j + o];
      a[j] = keep + __shfl_xor_sync(0xffffffffu, send, o);
    }
  }
  return a[0];
}

template <int MT, int COLS>  // rows of x and columns at a time
__global__ void __launch_bounds__(SF_THREADS, 2)
linear_stream_f32_kernel(const float* __restrict__ x, const float* __restrict__ w, void* __restrict__ out, int out_dtype, int M, int N, int K,
                         int ldo, float* __restrict__ partial, const float* __restrict__ bias) {
  pdl_launch_dependents();
  extern __shared__ __align__(16) float sf[];
  constexpr int D = sf_stages(MT, COLS);
  float* xs = sf;  // [MT][SF_KC]
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const unsigned ring = (unsigned)__cvta_generic_to_shared(sf + MT * SF_KC) + tid * 16;
  constexpr unsigned SLOT = SF_THREADS * 16, STAGE = SLOT * COLS;
  const int k0 = blockIdx.y * SF_KC, kn = min(SF_KC, K - k0), pieces = (kn + 127) / 128;
  // this warp's run of columns: the runs of all warps differ by one column at most
  const long long at = (long long)blockIdx.x * SF_WARPS + warp, all = (long long)gridDim.x * SF_WARPS;
  const int c0 = (int)(at * N / all), c1 = (int)((at + 1) * N / all);
  const float* wk = w + k0 + lane * 4;

  for (int m0 = 0; m0 < M; m0 += MT) {
    const int mt = min(MT, M - m0);
    int fc = c0, fp = 0;  // what is asked for next: columns from fc on, piece fp of the inner dimension
    auto fetch = [&](int stage) {
      if (fc < c1) {
        const bool inside = fp * 128 + lane * 4 < kn;
#pragma unroll
        for (int c = 0; c < COLS; ++c) {
          const bool live = inside && fc + c < c1;
          asm volatile("cp.async.cg.shared.global.L2::256B [%0], [%1], 16, %2;" ::"r"(ring + stage * STAGE + c * SLOT),
                       "l"(live ? wk + (size_t)(fc + c) * K + fp * 128 : w), "r"(live ? 16 : 0) : "memory");
        }
        if (++fp == pieces) {
          fp = 0;
          fc += COLS;
        }
      }
      asm volatile("cp.async.commit_group;" ::: "memory");
    };
    int stage = 0;
    for (; stage < D - 1; ++stage) fetch(stage);  // the weights do not depend on the kernel before this one
    if (m0 == 0) pdl_wait();
    else __syncthreads();  // the rows before these have been used by every warp
    for (int i = 0; i < MT; ++i)  // (rows there are not count as zeros: a branch per row would keep their loads apart)
      for (int k = tid * 4; k < kn; k += SF_THREADS * 4)
        *reinterpret_cast<float4*>(xs + i * SF_KC + k) =
            i < mt ? __ldg(reinterpret_cast<const float4*>(x + (size_t)(m0 + i) * K + k0 + k)) : make_float4(0.f, 0.f, 0.f, 0.f);
    __syncthreads();
    int src = 0;
    for (int n0 = c0; n0 < c1; n0 += COLS) {
      float acc[MT * COLS];  // [row][column]
#pragma unroll
      for (int i = 0; i < MT * COLS; ++i) acc[i] = 0.f;
      for (int p = 0; p < pieces; ++p) {
        asm volatile("cp.async.wait_group %0;" ::"n"(D - 2) : "memory");  // the oldest stage has landed
        fetch(stage);  // into the one that was used a turn ago
        stage = stage + 1 == D ? 0 : stage + 1;
        float4 v[COLS];
#pragma unroll
        for (int c = 0; c < COLS; ++c)
          asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
                       : "=f"(v[c].x), "=f"(v[c].y), "=f"(v[c].z), "=f"(v[c].w) : "r"(ring + src * STAGE + c * SLOT) : "memory");
        src = src + 1 == D ? 0 : src + 1;
        const int k = p * 128 + lane * 4;
        if (k < kn) {
#pragma unroll
          for (int i = 0; i < MT; ++i) {
            const float4 u = *reinterpret_cast<const float4*>(xs + i * SF_KC + k);
#pragma unroll
            for (int c = 0; c < COLS; ++c) {
              float t = acc[i * COLS + c];
              t = fmaf(v[c].x, u.x, t); t = fmaf(v[c].y, u.y, t); t = fmaf(v[c].z, u.z, t); t = fmaf(v[c].w, u.w, t);
              acc[i * COLS + c] = t;
            }
          }
        }
      }
      float v;
      if (MT * COLS == 32) {
        v = warp_sums_of_32(acc, lane);  // lane l ends up with sum l
      } else {
        v = 0.f;
#pragma unroll
        for (int i = 0; i < MT * COLS; ++i) {
          const float t = warp_sum(acc[i]);
          if (lane == i) v = t;
        }
      }
      const int i = lane / COLS, n = n0 + lane % COLS;
      if (i < mt && n < c1) {
        if (gridDim.y > 1) partial[((size_t)blockIdx.y * M + m0 + i) * N + n] = v;
        else store_from_f32(out, out_dtype, (size_t)(m0 + i) * ldo + n, bias ? v + bias[n] : v);
      }
    }
  }
}

// out[m, n] = partial[0][m, n] + partial[1][m, n] + ... in that order.
__global__ void __launch_bounds__(256)
linear_skinny_sum_kernel(const float* __restrict__ partial, int splits, void* __restrict__ out, int out_dtype, int M, int N, int ldo,
                         const float* __restrict__ bias) {
  pdl_launch_dependents();
  pdl_wait();
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= (size_t)M * N) return;
  const int m = (int)(i / N), n = (int)(i - (size_t)m * N);
  float v = 0.f;
  for (int s = 0; s < splits; ++s) v += partial[(size_t)s * M * N + i];
  if (bias) v += bias[n];
  store_from_f32(out, out_dtype, (size_t)m * ldo + n, v);
}

static int sk_sm_count() {
  static int n = 0;
  if (!n) {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0)
      n = 148;
  }
  return n;
}
// Over how many blocks the inner dimension of an [N, K] matrix is shared out.  float32: one per SF_KC elements.  bfloat16: enough for
// about four blocks per SM, at most one per chunk of x, and among those counts the one whose longest share
// of chunks is shortest.
extern "C" int bn_linear_skinny_splits(int N, int K, int dtype) {
  if (N <= 0 || K <= 0) return 1;
  if (dtype == BN_F32) return (K + SF_KC - 1) / SF_KC;
  const int blocks = (N + SK_WARPS * SK_COLS - 1) / (SK_WARPS * SK_COLS), chunks = (K + SK_KC - 1) / SK_KC;
  int want = (4 * sk_sm_count() + blocks - 1) / blocks;
  if (want > chunks) want = chunks;
  if (want <= 1) return 1;
  int best = want;
  for (int s = want; s <= chunks && s <= 2 * want; ++s)
    if ((chunks + s - 1) / s < (chunks + best - 1) / best) best = s;
  return best;
}

// x and w share the element type `dtype`; K must be a multiple of 8 (16-byte rows).  partial: float32
// scratch of bn_linear_skinny_splits(N, K, dtype) * M * N floats (not used when that is 1).  bias: [N] float32 added to every row, or
// null.
extern "C" int bn_linear_skinny(const void* x, const void* w, int dtype, void* out, int out_dtype, int M, int N,
                                int K, int ldo, float* partial, const float* bias, cudaStream_t stream) {
  if (M <= 0 || N <= 0) return BN_OK;
  if (K <= 0 || K % 8 || ldo < N) return BN_ERR_BAD_ARG;
  const int splits = bn_linear_skinny_splits(N, K, dtype);
  if ((splits > 1 && !partial) || splits > 65535) return BN_ERR_BAD_ARG;
  dim3 grid((unsigned)((N + SK_WARPS * SK_COLS - 1) / (SK_WARPS * SK_COLS)), (unsigned)splits);
  if (dtype == BN_F32) {
    // two blocks per SM in all, and of a small matrix a column per warp at least.  Four columns at a time, or so many fewer that a
    // warp's columns leave fewer places of its ring empty (8 rows: 6144 x 4096, up to six columns a warp, 34 us by twos and 37 by
    // fours; 4096 x 4096, up to four, 20 by fours and 23 by twos).
    unsigned columns = (unsigned)((N + SF_WARPS - 1) / SF_WARPS), most = (unsigned)(2 * sk_sm_count() / splits);
    if (most < 1) most = 1;
    grid.x = columns < most ? columns : most;
    const int per_warp = (N + (int)(grid.x * SF_WARPS) - 1) / (int)(grid.x * SF_WARPS);
#define SF_LAUNCH(MT, COLS)                                                                                                   \
  do {                                                                                                                        \
    static BnGrant grant;                                                                                                     \
    cudaError_t e = grant.ask((const void*)linear_stream_f32_kernel<MT, COLS>, sf_smem(MT), 0);                               \
    if (e != cudaSuccess) return BN_ERR_LAUNCH + (int)e;                                                                      \
    BN_LAUNCH((linear_stream_f32_kernel<MT, COLS>), grid, SF_THREADS, sf_smem(MT), stream, (const float*)x, (const float*)w,  \
              out, out_dtype, M, N, K, ldo, partial, bias);                                                                   \
  } while (0)
#define SF_COLUMNS(MT)                                                          \
  do {                                                                          \
    if (per_warp == 1) SF_LAUNCH(MT, 1);                                        \
    else if (per_warp == 2 || per_warp == 5 || per_warp == 6) SF_LAUNCH(MT, 2); \
    else SF_LAUNCH(MT, 4);                                                      \
  } while (0)
    if (M <= 2) SF_COLUMNS(2);
    else if (M <= 4) SF_COLUMNS(4);
    else SF_COLUMNS(8);
#undef SF_COLUMNS
#undef SF_LAUNCH
  } else if (dtype == BN_BF16)
    BN_LAUNCH((linear_skinny_kernel<__nv_bfloat16>), grid, SK_WARPS * 32, 0, stream,
              (const __nv_bfloat16*)x, (const __nv_bfloat16*)w, out, out_dtype, M, N, K, ldo, partial, bias);
  else
    return BN_ERR_BAD_ARG;
  if (splits > 1) {
    const size_t total = (size_t)M * N;
    BN_LAUNCH(linear_skinny_sum_kernel, (unsigned)((total + 255) / 256), 256, 0, stream, (const float*)partial, splits, out,
              out_dtype, M, N, ldo, bias);
  }
  BN_CHECK_LAUNCH();
  return BN_OK;
}
