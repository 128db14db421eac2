// out[M, N] = x[M, K] . W[N, K]^T in bfloat16 for M <= 16 and matrices that fit on the chip: a block has the whole of its 16 rows of W in shared
// memory before its input is there.
//
// Products of a few million weights are bound by what lies between them, not by their bytes: 2048 x 2048 are 1.3 us of memory time, but took
// 5 to 6 us in linear_tc.cu, whose tiles of 128 rows have to be shared out over clusters (TMA, one thread's MMAs, tensor memory, an
// exchange through the cluster's shared memories: each a round trip behind the other).  Here a block owns 16 rows and its eight warps share
// out the inner dimension.  Lanes copy their pieces of the weights into slots of their own as soon as the block starts, while the kernels
// before this one still run (programmatic dependent launch; several small products may be resident at once).  Behind the wait are one
// round of loads for the rows of x, mma.sync (weights as the 16 rows, tokens as the 8 columns; a lane's 16-byte pieces are at once its
// operands of two m16n8k16, since the order of the inner dimension is free as long as both operands take the same one), one exchange
// between the warps in shared memory, and the epilogue.  In a chain of dependent products of 2048 x 2048 one with 8 rows of x takes 1.9 us
// less than in linear_tc.cu, of 3072 x 2048 2.5, of 512 x 1024 2.5, of 64 x 256 2.0.
//
// Epilogues and arguments are those of linear_tc.cu: (0) store, with a bias or the square of the positive part; (2) gated unit over
// rows that alternate 8 gate and 8 up rows; (3) add to a float32 residual and prepare the RMSNorm that follows: residual * gain in bfloat16
// and the block's sum of squares per row; input rows that still lack their norm's scale (row_ss) have it applied to the result.
//
// Reference for the operation: y = W x with float32 accumulation (src/quant/bf16_scalar.c:4-21).
#include "common.cuh"
#include "mma.cuh"

#define LR_ROWS 16
#define LR_WARPS 8
#define LR_THREADS (32 * LR_WARPS)
#define LR_MAX_TOKENS 16
#define LR_BATCH 8  // pieces of x that a lane asks for at once, per group of tokens

struct LrArgs {
  const __nv_bfloat16 *x, *w;
  void* out;
  int out_dtype;
  int M, N, K, ldo, mode, act, groups;  // groups: pieces of 32 numbers of the inner dimension per warp
  const float* row_ss;
  int ss_parts, ss_stride;
  float inv_width, eps;
  const void* gain;
  int gain_dtype;
  __nv_bfloat16* xg;
  float* ss_out;
  int ss_out_stride;
};

template <int TG>  // groups of 8 tokens
__global__ void __launch_bounds__(LR_THREADS) linear_resident_kernel(LrArgs a) {
  pdl_launch_dependents();
  extern __shared__ __align__(16) uint4 lr_slots[];  // [groups][2][threads]
  __shared__ float4 parts[LR_WARPS][TG][32];
  __shared__ float ss_chunk[LR_THREADS], row_scale[8 * TG];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, quad = lane & 3;
  const int n0 = blockIdx.x * LR_ROWS, k0 = warp * a.groups * 32 + quad * 8;
  {
    const __nv_bfloat16* w0 = a.w + (size_t)(n0 + g) * a.K + k0;
    const bool row0 = n0 + g < a.N, row1 = n0 + g + 8 < a.N;
    const unsigned slot = (unsigned)__cvta_generic_to_shared(lr_slots) + tid * 16;
    for (int i = 0; i < a.groups; ++i) {
      const bool in = k0 + i * 32 < a.K;
      const int b0 = in && row0 ? 16 : 0, b1 = in && row1 ? 16 : 0;  // 0: zeros, the address is not read
      asm volatile("cp.async.cg.shared.global.L2::256B [%0], [%1], 16, %2;" ::"r"(slot + (2 * i) * (LR_THREADS * 16)),
                   "l"(b0 ? w0 + i * 32 : a.w), "r"(b0) : "memory");
      asm volatile("cp.async.cg.shared.global.L2::256B [%0], [%1], 16, %2;" ::"r"(slot + (2 * i + 1) * (LR_THREADS * 16)),
                   "l"(b1 ? w0 + (size_t)8 * a.K + i * 32 : a.w), "r"(b1) : "memory");
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
  pdl_wait();
  // what does not depend on the products is asked for first: sums of squares of the input rows, the residual and the gains
  float ss = 0.f;
  if (a.row_ss != nullptr) {
    constexpr int CH = LR_THREADS / (8 * TG);
    const int m = tid % (8 * TG), c = tid / (8 * TG), per = (a.ss_parts + CH - 1) / CH;
    if (m < a.M)
      for (int p = c * per; p < min(a.ss_parts, (c + 1) * per); ++p) ss += a.row_ss[(size_t)p * a.ss_stride + m];
  }
  // an item of the epilogue: row r of the block, token m
  const int r = tid & (LR_ROWS - 1), m = tid >> 4, n = n0 + r;
  const bool live = m < a.M && n < a.N;
  float gain = 0.f, old = 0.f;
  if (a.mode != 2 && live && a.gain != nullptr) gain = load_as_f32(a.gain, a.gain_dtype, (size_t)n);
  if (a.mode == 3 && live) old = ((const float*)a.out)[(size_t)m * a.ldo + n];

  float acc[TG][4];
#pragma unroll
  for (int t = 0; t < TG; ++t) acc[t][0] = acc[t][1] = acc[t][2] = acc[t][3] = 0.f;
  for (int i0 = 0; i0 < a.groups; i0 += LR_BATCH) {
    uint4 xv[LR_BATCH][TG];
#pragma unroll
    for (int i = 0; i < LR_BATCH; ++i)
#pragma unroll
      for (int t = 0; t < TG; ++t) {
        const int k = k0 + (i0 + i) * 32, tok = t * 8 + g;
        xv[i][t] = make_uint4(0u, 0u, 0u, 0u);
        if (i0 + i < a.groups && k < a.K && tok < a.M) xv[i][t] = *reinterpret_cast<const uint4*>(a.x + (size_t)tok * a.K + k);
      }
    if (i0 == 0) asm volatile("cp.async.wait_group 0;" ::: "memory");  // this lane's own pieces: nobody else reads them
#pragma unroll
    for (int i = 0; i < LR_BATCH; ++i)
      if (i0 + i < a.groups) {
        const uint4 w0 = lr_slots[(2 * (i0 + i)) * LR_THREADS + tid], w1 = lr_slots[(2 * (i0 + i) + 1) * LR_THREADS + tid];
#pragma unroll
        for (int t = 0; t < TG; ++t) {
          mma_bf16(acc[t], w0.x, w1.x, w0.y, w1.y, xv[i][t].x, xv[i][t].y);
          mma_bf16(acc[t], w0.z, w1.z, w0.w, w1.w, xv[i][t].z, xv[i][t].w);
        }
      }
  }
#pragma unroll
  for (int t = 0; t < TG; ++t) parts[warp][t][lane] = make_float4(acc[t][0], acc[t][1], acc[t][2], acc[t][3]);
  ss_chunk[tid] = ss;
  __syncthreads();
  if (a.row_ss != nullptr) {
    constexpr int CH = LR_THREADS / (8 * TG);
    if (tid < a.M) {
      float tot = 0.f;
      for (int c = 0; c < CH; ++c) tot += ss_chunk[c * 8 * TG + tid];
      row_scale[tid] = 1.0f / sqrtf(tot * a.inv_width + a.eps);
    }
    __syncthreads();
  }
  // lane 4 g + q of a warp holds rows g and g + 8 of tokens 2 q and 2 q + 1
  auto value = [&](int row, int tok) {
    const float* p = &parts[0][tok >> 3][(row & 7) * 4 + ((tok & 7) >> 1)].x + (row >> 3) * 2 + (tok & 1);
    float v = 0.f;
#pragma unroll
    for (int w = 0; w < LR_WARPS; ++w) v += p[w * TG * 128];
    return a.row_ss != nullptr ? v * row_scale[tok] : v;
  };
  if (a.mode == 2) {
    const int j = tid & 7, tok = tid >> 3;
    if (tok < a.M && n0 + j < a.N) {
      const float gv = value(j, tok), uv = value(j + 8, tok);
      store_from_f32(a.out, a.out_dtype, (size_t)tok * a.ldo + (n0 >> 1) + j,
                     (a.act == BN_ACT_SILU ? __fdividef(gv, 1.0f + __expf(-gv)) : glu_activation(gv, a.act)) * uv);
    }
    return;
  }
  if (a.mode == 0) {
    if (live) {
      float y = value(r, m) + gain;  // the bias, or zero
      if (a.act == BN_ACT_RELU2) y = relu_squared(y);
      store_from_f32(a.out, a.out_dtype, (size_t)m * a.ldo + n, y);
    }
    return;
  }
  float sq = 0.f;
  if (live) {
    const float nv = old + value(r, m);
    ((float*)a.out)[(size_t)m * a.ldo + n] = nv;
    a.xg[(size_t)m * a.N + n] = __float2bfloat16_rn(nv * gain);
    sq = nv * nv;
  }
#pragma unroll
  for (int o = LR_ROWS / 2; o > 0; o >>= 1) sq += __shfl_xor_sync(0xffffffffu, sq, o);
  if (r == 0 && m < a.M) a.ss_out[(size_t)blockIdx.x * a.ss_out_stride + m] = sq;
}

// x [M, K], w [N, K] bfloat16, 16-byte aligned with K a multiple of 8; modes, gain, xg, ss_out and row_ss as bn_linear_tc_ex has them
// (ss_out: a part per 16 rows of w).  M up to 16; a block's rows of w must fit its shared memory (K up to 6,144).
extern "C" int bn_linear_resident(const void* x, const void* w, void* out, int out_dtype, int M, int N, int K, int ldo, int mode,
                                  const float* row_ss, int ss_parts, int ss_stride, float inv_width, float eps, const void* gain, int gain_dtype,
                                  void* xg, float* ss_out, int ss_out_stride, cudaStream_t stream) {
  if (M <= 0 || N <= 0) return BN_OK;
  const int act = mode >> 8;
  mode &= 255;
  if (act != BN_ACT_SILU && act != BN_ACT_GELU_TANH && !(act == BN_ACT_RELU2 && mode == 0)) return BN_ERR_BAD_ARG;
  if (!x || !w || !out || M > LR_MAX_TOKENS || K <= 0 || K % 8 || K > 6144 || (mode != 0 && mode != 2 && mode != 3)) return BN_ERR_BAD_ARG;
  if (mode == 2 && (N % 16)) return BN_ERR_BAD_ARG;
  if (mode == 3 && (!gain || !xg || !ss_out || ss_out_stride < M || out_dtype != BN_F32)) return BN_ERR_BAD_ARG;
  if (mode != 2 && gain && gain_dtype != BN_F32 && gain_dtype != BN_BF16) return BN_ERR_BAD_ARG;
  if (row_ss && (ss_parts <= 0 || ss_stride < M)) return BN_ERR_BAD_ARG;
  if (((uintptr_t)x | (uintptr_t)w) & 15) return BN_ERR_BAD_ARG;
  LrArgs a;
  a.x = (const __nv_bfloat16*)x; a.w = (const __nv_bfloat16*)w; a.out = out; a.out_dtype = out_dtype;
  a.M = M; a.N = N; a.K = K; a.ldo = ldo; a.mode = mode; a.act = act;
  a.groups = (K + 32 * LR_WARPS - 1) / (32 * LR_WARPS);
  a.row_ss = row_ss; a.ss_parts = ss_parts; a.ss_stride = ss_stride; a.inv_width = inv_width; a.eps = eps;
  a.gain = gain; a.gain_dtype = gain_dtype; a.xg = (__nv_bfloat16*)xg; a.ss_out = ss_out; a.ss_out_stride = ss_out_stride;
  const size_t smem = (size_t)a.groups * 2 * LR_THREADS * 16;
  const unsigned grid = (unsigned)((N + LR_ROWS - 1) / LR_ROWS);
#define LR_RUN(TG)                                                                       \
  do {                                                                                   \
    static BnGrant grant;                                                                \
    cudaError_t e = grant.ask((const void*)linear_resident_kernel<TG>, smem, 10 * 1024); \
    if (e != cudaSuccess) return BN_ERR_LAUNCH + (int)e;                                 \
    BN_LAUNCH((linear_resident_kernel<TG>), grid, LR_THREADS, smem, stream, a);          \
  } while (0)
  if (M <= 8) LR_RUN(1);
  else LR_RUN(2);
  BN_CHECK_LAUNCH();
  return BN_OK;
}
