// out[M, N] = x[M, K] . W[N, K]^T (+ a bias) in float32 for many rows, on the 5th-generation tensor cores (tcgen05).
//
// A float32 number is the sum of three bfloat16 numbers, exactly: its leading eight bits, the next eight, and what is left, at most eight bits.
// x's are rounded, W's cut off: beside the power of two at or below a number, x's middle and low parts are at most 2^-8 and 2^-17, W's less than
// 2^-7 and 2^-15.  Of the nine products of two such sums six are kept (high x high, the two of high x middle, middle x middle, the two of
// high x low); the other three come to less than 2^-24 + 2^-23 + 2^-32 of the product, with signs of their own.  The tensor cores multiply
// exactly and add up in their accumulator, which cuts off where an addition rounds, so a sum stays there for 32 numbers of the inner
// dimension only (small products first) and is then added in float32: the error against 64 bits is a third to a sixth of the float32 library
// product's (520 rows, 4096 x 4096: 2.2e-7 against 1.1e-6 of the result's norm; 1024 x 14336: 3.9e-7 against 2.2e-6).
//
// The float32 units reach 72 TFLOP/s at most, the library's product 54; six bfloat16 products per float32 product are 230 TFLOP/s at the tensor
// cores' rate.  520 rows: 28672 x 4096 611 us (library 2289), 6144 x 4096 129 (540), 4096 x 4096 109 (325), 4096 x 14336 356 (1126); scaling W on the way
// (below) takes 0 to 2 % of that: 28672 x 4096 behind a flush of the L2 617 -> 620.
//
// A tile is 128 rows of W times up to 192 rows of x: D[128 rows of W, NT rows of x], so that few and odd numbers of rows of x waste
// little (NT is a multiple of 16, chosen so that the tiles fill the SMs).  x is split once, by a kernel of its own, into three
// planes of bfloat16 in memory (it is small, and every tile column of W reads it again).  W is split on the way: its float32 tiles arrive by
// TMA, groups of four warps turn a row each thread into three bfloat16 operands in tensor memory, from where the MMA takes its A operand; in
// shared memory they would cost more of its bandwidth than there is (the MMAs read 5.6 KB of x's planes in 88 cycles each).
//
// A persistent block of 20 warps per SM:
//   warp 0      requests float32 tiles of W (128 rows x 32 numbers)
//   warp 1      requests tiles of x's three planes (NT rows x 32 numbers each, 64-byte swizzle)
//   warp 2      allocates tensor memory; issues twelve MMAs per 32 numbers, into one of two accumulators
//   warps 4-11  split W: shared memory -> registers -> tensor memory, two groups of four warps with a buffer each take turns
//   warps 12-19 add the accumulators up in registers (a row of W each thread, two warps share a row's columns) and store
//
// Three bfloat16 numbers hold a float32 only while the last of them is no subnormal number (below 2^-109 bits were lost), so both operands are
// scaled by 2^24 first, which takes float32's smallest numbers there, and the sums are scaled back.  Products and sums stay finite while
// numbers are below 2^30; a row of x with a larger one has a smaller scale of its own.  What does not split (rows of x with numbers that are not
// finite, or so far apart that the smallest lose bits; rows of W with a number of 2^30 or more, or not finite) is marked, of x by the kernel
// that splits it, of W by the warps that do, and outputs of marked rows are computed again in plain float32 by the warps that add, four rows of W times four of x at a
// time (520 rows, 4096 x 4096, 131 us: with one marked row of W 582, of x 283, with all rows marked 2,660; a thread per output took 14,700, 600 and
// 69,000.  The other warps wait meanwhile: for a tile whose rows are all marked some 3 ms at K = 4,096, 0.2 s of their limit of 2 s at the largest K).
//
// The twelve MMAs of 32 numbers take 1,060 cycles for 176 rows of x; a wait for an mbarrier costs its role some 200, even if it is over.  So
// the whole of warp 2 walks its loop, with descriptors in uniform registers, and one elected lane issues (as one thread's work a step took 1,700
// cycles: 790 to issue, 900 for three waits).  Splitting 32 numbers of a row, which is a chain of waits, loads and stores, takes a warp 1,400: so
// two groups take turns (with one 4096 x 4096 117 us, 128 rows of 6144 x 4096 108 instead of 73; before both 133 and 28672 x 4096 705).
//
// The adding warps keep 96 sums a thread in registers.  The block starts with 96 registers for each of 640 threads, and its warps share them
// anew: 4 x 40 + 8 x 88 + 8 x 128 = 1,888 of 20 x 96 = 1,920 per lane, so that nobody waits for registers.
//
// Every wait on an mbarrier is bounded in time; a wait that gives up records code 8 in *status, every role leaves its loops (the others
// when a wait of theirs gives up in turn), and the block frees its tensor memory and returns.
//
// Reference: y = W x with float32 accumulation (src/quant/f32_scalar.c:4-32); the reference's CUDA prefill calls cublasSgemm
// (src/gpu_cuda.cu:11788-11879).
#include "tma.cuh"
#include "umma.cuh"

#define LS_BM 128        // rows of W per tile (UMMA M)
#define LS_BK 32         // numbers of the inner dimension per stage and per sum in the tensor cores
#define LS_NT_MAX 192    // rows of x per tile at most
#define LS_THREADS 640   // five warpgroups
#define LS_W_STAGES 4
#define LS_W_BYTES (LS_BM * LS_BK * 4)
#define LS_X_STAGES_MAX 8
#define LS_A_COLS 48     // columns of tensor memory per buffer of W's three operands (two numbers a column)
#define LS_ACC_COLS LS_NT_MAX
#define LS_SMEM_MAX (224 * 1024)
#define LS_ERR_WAIT 8

struct LsArgs {
  float* out;
  const float *x, *w, *bias;
  const float* x_unscale;  // [M] what takes a sum back to x's and W's own scale; 0: a marked row
  int M, N, K, ldo, k_blocks;
  int nt, m_tiles, n_tiles, x_stages;
  int* status;
};

// Two numbers as three pairs of bfloat16, rounded
__device__ __forceinline__ void ls_split(float a, float b, unsigned& high, unsigned& mid, unsigned& low) {
  high = pack_bf16x2(a, b);
  const float ra = a - __uint_as_float(high << 16), rb = b - __uint_as_float(high & 0xffff0000u);
  mid = pack_bf16x2(ra, rb);
  low = pack_bf16x2(ra - __uint_as_float(mid << 16), rb - __uint_as_float(mid & 0xffff0000u));
}
// The same cut off instead of rounded, which takes no conversions.  The signs of what the products leave out follow x's parts, which are
// rounded to either side.
__device__ __forceinline__ void ls_cut(float a, float b, unsigned& high, unsigned& mid, unsigned& low) {
  const unsigned ua = __float_as_uint(a), ub = __float_as_uint(b);
  high = __byte_perm(ua, ub, 0x7632);
  const float ra = a - __uint_as_float(ua & 0xffff0000u), rb = b - __uint_as_float(ub & 0xffff0000u);
  const unsigned va = __float_as_uint(ra), vb = __float_as_uint(rb);
  mid = __byte_perm(va, vb, 0x7632);
  low = __byte_perm(__float_as_uint(ra - __uint_as_float(va & 0xffff0000u)), __float_as_uint(rb - __uint_as_float(vb & 0xffff0000u)), 0x7632);
}
#define LS_SCALE 16777216.0f  // 2^24
#define LS_LARGE 1073741824.0f  // 2^30
#define LS_MARK 316912650057057350374175801344.0f  // 2^98: LS_LARGE times it is infinite
#define LS_MAX_K (1 << 18)  // products below 2^54 2^54, so many of them below 2^127
__device__ __forceinline__ float ls_power(int e) { return __uint_as_float((unsigned)(e + 127) << 23); }  // 2^e, a normal number

// planes [3][M][pitch] bfloat16 and the scales of x [M, K]; a block per row
__global__ void __launch_bounds__(256) linear_split_rows_kernel(const float* __restrict__ x, int M, int K, int pitch, __nv_bfloat16* __restrict__ planes,
                                                                 float* __restrict__ unscale) {
  pdl_wait();
  pdl_launch_dependents();  // (not before: the product's blocks read W without a wait of their own, and the kernel in front may have written it)
  __shared__ unsigned s_most[8];
  const int m = blockIdx.x;
  const float* row = x + (size_t)m * K;
  const size_t plane = (size_t)M * pitch;
  __nv_bfloat16* to = planes + (size_t)m * pitch;
  unsigned most = 0;  // (sizes of numbers are in the order of their bits, behind them infinities and what is not a number)
  bool lost = false;
  auto rows = [&](float scale, auto look) {
    for (int k = threadIdx.x * 4; k < K; k += 1024) {  // K is a multiple of 4
      const float4 v = *reinterpret_cast<const float4*>(row + k);
      const float a = v.x * scale, b = v.y * scale, c = v.z * scale, d = v.w * scale;
      uint2 h, i, l;
      ls_split(a, b, h.x, i.x, l.x);
      ls_split(c, d, h.y, i.y, l.y);
      *reinterpret_cast<uint2*>(to + k) = h;
      *reinterpret_cast<uint2*>(to + plane + k) = i;
      *reinterpret_cast<uint2*>(to + 2 * plane + k) = l;
      look(v, h, i, l);
    }
  };
  rows(LS_SCALE, [&](float4 v, uint2, uint2, uint2) {
    const unsigned ab = max(__float_as_uint(v.x) & 0x7fffffffu, __float_as_uint(v.y) & 0x7fffffffu);
    most = max(max(most, ab), max(__float_as_uint(v.z) & 0x7fffffffu, __float_as_uint(v.w) & 0x7fffffffu));
  });
  if (!__syncthreads_or(most >= __float_as_uint(LS_LARGE))) {
    if (threadIdx.x == 0) unscale[m] = 1.0f / (LS_SCALE * LS_SCALE);
    return;
  }
  // a row with large numbers: its largest goes to [2^53, 2^54)
  most = __reduce_max_sync(0xffffffffu, most);
  if ((threadIdx.x & 31) == 0) s_most[threadIdx.x >> 5] = most;
  __syncthreads();
  for (int i = 0; i < 8; ++i) most = max(most, s_most[i]);
  if (most >= 0x7f800000u) {
    if (threadIdx.x == 0) unscale[m] = 0.f;
    return;
  }
  const int e = 53 - ((int)(most >> 23) - 127);
  const float back = ls_power(-e);
  rows(ls_power(e), [&](float4 v, uint2 h, uint2 i, uint2 l) {
    auto whole = [&](float one, unsigned high, unsigned mid, unsigned low, bool upper) {  // whether the parts add up to the number
      auto part = [&](unsigned p) { return __uint_as_float(upper ? p & 0xffff0000u : p << 16); };
      return ((part(high) + part(mid)) + part(low)) * back == one;
    };
    lost |= !(whole(v.x, h.x, i.x, l.x, false) & whole(v.y, h.x, i.x, l.x, true) & whole(v.z, h.y, i.y, l.y, false) & whole(v.w, h.y, i.y, l.y, true));
  });
  lost = __syncthreads_or(lost);
  if (threadIdx.x == 0) unscale[m] = lost ? 0.f : back * (1.0f / LS_SCALE);
}

// K-major tile with rows of 64 bytes, 64-byte swizzled: groups of 8 rows 512 bytes apart
__device__ __forceinline__ unsigned long long ls_desc(unsigned addr) {
  return (unsigned long long)((addr >> 4) & 0x3FFF) | (1ull << 16) | (32ull << 32) | (1ull << 46) | (4ull << 61);
}
// The outputs of marked rows among rows n0 .. n0 + 31 of W (bit i of `rows`: n0 + i is marked) and m0 .. m_end - 1 of x, in plain float32: a warp takes
// four by four at a time, its lanes share the inner dimension.
__device__ __noinline__ void ls_plain(const LsArgs& a, unsigned rows, int n0, int m0, int m_end, int lane) {
  for (int m = m0; m < m_end; m += 4) {
    unsigned cols = 0;
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (m + j < m_end && a.x_unscale[m + j] == 0.f) cols |= 1u << j;
    for (int i0 = 0; i0 < 32 && n0 + i0 < a.N; i0 += 4) {
      const unsigned some = (rows >> i0) & 15u;
      if ((some | cols) == 0) continue;
      const float *w[4], *x[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        w[i] = a.w + (size_t)min(n0 + i0 + i, a.N - 1) * a.K;
        x[i] = a.x + (size_t)min(m + i, m_end - 1) * a.K;
      }
      float sum[16];
#pragma unroll
      for (int i = 0; i < 16; ++i) sum[i] = 0.f;
      for (int k = lane * 4; k < a.K; k += 128) {
        float4 wv[4], xv[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          wv[i] = *reinterpret_cast<const float4*>(w[i] + k);
          xv[i] = *reinterpret_cast<const float4*>(x[i] + k);
        }
#pragma unroll
        for (int i = 0; i < 16; ++i)
          sum[i] = fmaf(wv[i >> 2].x, xv[i & 3].x, fmaf(wv[i >> 2].y, xv[i & 3].y, fmaf(wv[i >> 2].z, xv[i & 3].z, fmaf(wv[i >> 2].w, xv[i & 3].w, sum[i]))));
      }
      float mine = 0.f;
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        const float s = warp_sum(sum[i]);
        if (lane == i) mine = s;
      }
      const int i = lane >> 2, j = lane & 3, n = n0 + i0 + i;
      if (lane < 16 && ((some >> i | cols >> j) & 1u) && n < a.N && m + j < m_end)
        a.out[(size_t)(m + j) * a.ldo + n] = mine + (a.bias != nullptr ? a.bias[n] : 0.f);
    }
  }
}

template <int CH>  // an adding warp takes 16 CH columns, the tile has up to 32 CH
__global__ void __launch_bounds__(LS_THREADS, 1)
linear_split_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x, const __grid_constant__ LsArgs a) {
  pdl_launch_dependents();
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char* base = (unsigned char*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  const unsigned plane_bytes = a.nt * LS_BK * 2, x_bytes = 3 * plane_bytes;  // nt is a multiple of 16: whole 1024 bytes
  unsigned char* x_ring = base + LS_W_STAGES * LS_W_BYTES;
  __shared__ unsigned long long bars[2 * LS_W_STAGES + 2 * LS_X_STAGES_MAX + 7];
  __shared__ unsigned tmem_slot;
  __shared__ int s_failed;
  __shared__ unsigned char w_marked[2][2][LS_BM];  // by turn of the tile, group of splitting warps, row
  volatile int* failed = &s_failed;
  const unsigned w_full = smem_u32(bars), w_free = w_full + 8 * LS_W_STAGES, x_full = w_free + 8 * LS_W_STAGES, x_free = x_full + 8 * LS_X_STAGES_MAX,
                 a_full = x_free + 8 * LS_X_STAGES_MAX, acc_full = a_full + 16, acc_free = acc_full + 16, marks = acc_free + 16;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (tid == 0) {
    s_failed = 0;
    tma_prefetch_map(&map_w);
    tma_prefetch_map(&map_x);
    for (int s = 0; s < LS_W_STAGES; ++s) {
      mbar_init(w_full + 8 * s, 1);
      mbar_init(w_free + 8 * s, 4);
    }
    for (int s = 0; s < LS_X_STAGES_MAX; ++s) {
      mbar_init(x_full + 8 * s, 1);
      mbar_init(x_free + 8 * s, 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(a_full + 8 * b, 4);
      mbar_init(acc_full + 8 * b, 1);
      mbar_init(acc_free + 8 * b, 8);
    }
    mbar_init(marks, 8);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 2) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)), "r"(512u) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const unsigned tmem = tmem_slot;  // accumulators at 0 and LS_ACC_COLS, W's operands behind them
  const unsigned tmem_a = tmem + 2 * LS_ACC_COLS;
  const int tiles = a.m_tiles * a.n_tiles;
  // tile t: rows of W from (t / m_tiles) * 128, rows of x from (t % m_tiles) * nt (the blocks that run at once share rows of W)
  auto wait = [&](unsigned bar, unsigned parity) {
    if (mbar_wait(bar, parity & 1u, a.status, LS_ERR_WAIT)) return true;
    *failed = 1;  // (the other roles find out when a wait of theirs gives up)
    return false;
  };

  if (warp < 4) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 40;");
  }
  if (warp == 0) {
    if (lane == 0) {
      int s = 0, round = 0;
      bool ok = true;
      for (int t = blockIdx.x; ok && t < tiles; t += gridDim.x)
        for (int kb = 0; kb < a.k_blocks; ++kb) {
          if (round > 0 && !(ok = wait(w_free + 8 * s, round - 1))) break;
          mbar_expect_tx(w_full + 8 * s, LS_W_BYTES);
          tma_load_2d(smem_u32(base + s * LS_W_BYTES), &map_w, w_full + 8 * s, kb * LS_BK, t / a.m_tiles * LS_BM);
          if (++s == LS_W_STAGES) { s = 0; ++round; }
        }
    }
  } else if (warp == 1) {
    if (lane == 0) {
      pdl_wait();
      int s = 0, round = 0;
      bool ok = true;
      for (int t = blockIdx.x; ok && t < tiles; t += gridDim.x)
        for (int kb = 0; kb < a.k_blocks; ++kb) {
          if (round > 0 && !(ok = wait(x_free + 8 * s, round - 1))) break;
          mbar_expect_tx(x_full + 8 * s, x_bytes);
          for (int p = 0; p < 3; ++p)  // rows behind x's last are another plane's, or zeros: their results are not stored
            tma_load_2d(smem_u32(x_ring + s * x_bytes + p * plane_bytes), &map_x, x_full + 8 * s, kb * LS_BK, p * a.M + t % a.m_tiles * a.nt);
          if (++s == a.x_stages) { s = 0; ++round; }
        }
    }
  } else if (warp == 2) {
    // the whole warp walks the loop, so that addresses and descriptors are warp-uniform values
    const bool issuer = elect_one();
    const unsigned tbase = __shfl_sync(0xffffffffu, tmem, 0);
    // D float32, A and B bfloat16, both K-major, N >> 3 at bit 17, M >> 4 at bit 24
    const unsigned idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((unsigned)(a.nt >> 3) << 17) | ((LS_BM >> 4) << 24);
    const unsigned long long desc0 = ls_desc(smem_u32(x_ring));
    int s = 0, round = 0, it = 0;
    bool ok = true;
    for (int t = blockIdx.x; ok && t < tiles; t += gridDim.x)
      for (int kb = 0; kb < a.k_blocks; ++kb, ++it) {
        const int b = it & 1, use = it >> 1;
        // what is ready first is waited for first; W's operands are the last to come
        ok = __all_sync(0xffffffffu, (use == 0 || wait(acc_free + 8 * b, use - 1)) && wait(x_full + 8 * s, round) && wait(a_full + 8 * b, use));
        if (!ok) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        if (issuer) {
          const unsigned acc = tbase + b * LS_ACC_COLS, wa = tbase + 2 * LS_ACC_COLS + b * LS_A_COLS;
          const unsigned long long xd = desc0 + ((s * x_bytes) >> 4);
          const unsigned plane = plane_bytes >> 4;
          // planes of W and x (0 high, 1 middle, 2 low), the smallest products first
          constexpr int PW[6] = {2, 1, 0, 1, 0, 0}, PX[6] = {0, 1, 2, 0, 1, 0};
#pragma unroll
          for (int i = 0; i < 6; ++i)
#pragma unroll
            for (int kk = 0; kk < LS_BK / 16; ++kk)
              umma_mma_ts(acc, wa + PW[i] * 16 + kk * 8, xd + PX[i] * plane + kk * 2, idesc, (i | kk) ? 1u : 0u);
          umma_commit(x_free + 8 * s);   // arrives when these MMAs have read the stage
          umma_commit(acc_full + 8 * b);  // and W's operands, and the sums are complete
        }
        __syncwarp();
        if (++s == a.x_stages) { s = 0; ++round; }
      }
  } else if (warp >= 4 && warp < 12) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 88;");
    // group 0 splits the even steps' numbers into buffer 0, group 1 the odd steps' into buffer 1
    const int group = (warp - 4) >> 2, row = (warp & 3) * 32 + lane;
    const unsigned to = tmem_a + ((unsigned)((warp & 3) * 32) << 16) + group * LS_A_COLS;
    int kb = group, tile_i = 0, it = group;
    bool ok = true;
    float none = 0.f;
    for (int t = blockIdx.x; ok && t < tiles;) {
      const int s = it % LS_W_STAGES, use = it >> 1;
      ok = __all_sync(0xffffffffu, wait(w_full + 8 * s, it / LS_W_STAGES));
      if (!ok) break;
      const unsigned char* from = base + s * LS_W_BYTES + row * 128;
      float4 v[8];
#pragma unroll
      for (int c = 0; c < 8; ++c) v[c] = *reinterpret_cast<const float4*>(from + ((c ^ (row & 7)) << 4));
      unsigned high[16], mid[16], low[16];
#pragma unroll
      for (int c = 0; c < 8; ++c) {
        ls_cut(v[c].x * LS_SCALE, v[c].y * LS_SCALE, high[2 * c], mid[2 * c], low[2 * c]);
        ls_cut(v[c].z * LS_SCALE, v[c].w * LS_SCALE, high[2 * c + 1], mid[2 * c + 1], low[2 * c + 1]);
        // finite, until a number is 2^30 or more, or not finite (or their sum is: such a row is marked without need)
        none = fmaf(v[c].x, LS_MARK, fmaf(v[c].y, LS_MARK, fmaf(v[c].z, LS_MARK, fmaf(v[c].w, LS_MARK, none))));
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(w_free + 8 * s);
      if (use > 0) {  // the MMAs that read this buffer two steps ago are done
        ok = __all_sync(0xffffffffu, wait(acc_full + 8 * group, use - 1));
        if (!ok) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      }
      tmem_st16(to, reinterpret_cast<const float*>(high));
      tmem_st16(to + 16, reinterpret_cast<const float*>(mid));
      tmem_st16(to + 32, reinterpret_cast<const float*>(low));
      const bool last = kb + 2 >= a.k_blocks;  // this group's last step of the tile
      // (the adding warps have read the marks of two tiles before: a tile has at least four steps)
      if (last) w_marked[tile_i & 1][group][row] = !(fabsf(none) <= 3.402823466e38f);
      asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) {
        if (last) mbar_arrive(marks);
        mbar_arrive(a_full + 8 * group);
      }
      it += 2;
      kb += 2;
      if (last) {
        kb -= a.k_blocks;
        t += gridDim.x;
        ++tile_i;
        none = 0.f;
      }
    }
  } else if (warp >= 12) {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 128;");
    const int quad = warp & 3, row = quad * 32 + lane, c0 = ((warp - 12) >> 2) * 16 * CH;
    const unsigned from0 = tmem + ((unsigned)(quad * 32) << 16) + c0;
    int it = 0, tile_i = 0;
    bool ok = true, waited = false;
    for (int t = blockIdx.x; ok && t < tiles; t += gridDim.x, ++tile_i) {
      float acc[16 * CH];
#pragma unroll
      for (int c = 0; c < 16 * CH; ++c) acc[c] = 0.f;
      int row_marked = 0;
      for (int kb = 0; kb < a.k_blocks; ++kb, ++it) {
        const int b = it & 1, use = it >> 1;
        ok = __all_sync(0xffffffffu, wait(acc_full + 8 * b, use));
        if (!ok) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
        for (int j = 0; j < CH; ++j)
          if (c0 + j * 16 < a.nt) {
            float v[16];
            tmem_ld16(from0 + b * LS_ACC_COLS + j * 16, v);
#pragma unroll
            for (int c = 0; c < 16; ++c) acc[j * 16 + c] += v[c];
          }
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        if (kb + 1 == a.k_blocks) {
          ok = __all_sync(0xffffffffu, wait(marks, tile_i));
          if (!ok) break;
          row_marked = w_marked[tile_i & 1][0][row] | w_marked[tile_i & 1][1][row];
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(acc_free + 8 * b);
      }
      if (!ok) break;
      if (!waited) {
        pdl_wait();
        waited = true;
      }
      const int n = t / a.m_tiles * LS_BM + row, m0 = t % a.m_tiles * a.nt + c0, m_end = min(a.M, t % a.m_tiles * a.nt + a.nt);
      const float bias = n < a.N && a.bias != nullptr ? a.bias[n] : 0.f;
      bool plain = row_marked && n < a.N;
#pragma unroll
      for (int c = 0; c < 16 * CH; ++c) {
        const int m = m0 + c;
        if (m < m_end) {
          const float back = a.x_unscale[m];
          plain |= back == 0.f;
          if (n < a.N) a.out[(size_t)m * a.ldo + n] = fmaf(acc[c], back, bias);
        }
      }
      __syncwarp();  // (of two stores to one place the second one stays)
      if (__any_sync(0xffffffffu, plain)) ls_plain(a, __ballot_sync(0xffffffffu, row_marked), n - lane, m0, min(m_end, m0 + 16 * CH), lane);
    }
  }

  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (*failed) {
    // a wait gave up: loads that were requested may still be landing in this block's shared memory
    unsigned long long t0 = global_timer();
    while (global_timer() - t0 < 200000ull) __nanosleep(1000);
    __syncthreads();
  }
  if (warp == 2) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
  }
}

static int ls_sm_count() {
  static int n = 0;
  if (!n) {
    int dev = 0, v = 0;
    n = cudaGetDevice(&dev) == cudaSuccess && cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev) == cudaSuccess && v > 0 ? v : 148;
  }
  return n;
}

// A matrix [rows, cols] whose rows lie row_bytes apart, loaded in boxes of box_rows rows of 32 numbers (zeros outside).  Kind 3: float32,
// 128-byte swizzle; kind 4: bfloat16, 64-byte swizzle.
static bool ls_map(CUtensorMap* map, int kind, const void* ptr, unsigned long long rows, unsigned long long cols, unsigned long long row_bytes,
                   int box_rows) {
  if (tma_map_lookup(kind, ptr, rows, cols, row_bytes, box_rows, map)) return true;
  PFN_cuTensorMapEncodeTiled enc = tma_encoder();
  if (!enc) return false;
  cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows}, strides[1] = {(cuuint64_t)row_bytes};
  cuuint32_t box[2] = {LS_BK, (cuuint32_t)box_rows}, estr[2] = {1, 1};
  if (enc(map, kind == 3 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(ptr), dims, strides, box, estr,
          CU_TENSOR_MAP_INTERLEAVE_NONE, kind == 3 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
          CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
    return false;
  tma_map_keep(kind, ptr, rows, cols, row_bytes, box_rows, map);
  return true;
}

// Rows of x per tile: the number of tiles of rows for which the last wave costs least.  A tile costs its rows plus LS_TILE_COST.
#define LS_TILE_COST 24
static int ls_choose_nt(int M, int n_tiles, int sms) {
  const int least = (M + LS_NT_MAX - 1) / LS_NT_MAX;
  int best_nt = 0;
  long long best = 0;
  for (int mt = least; mt < least + 6; ++mt) {
    const int nt = ((M + mt - 1) / mt + 15) / 16 * 16;
    const long long tiles = (long long)n_tiles * ((M + nt - 1) / nt), cost = (tiles + sms - 1) / sms * (nt + LS_TILE_COST);
    if (best_nt == 0 || cost < best) { best = cost; best_nt = nt; }
    if (nt == 16) break;
  }
  return best_nt;
}

// Whether a block starts with as many registers as its warps share out (else a warp would wait for some that nobody gives back)
template <int CH>
static bool ls_registers() {
  static const bool enough = [] {
    cudaFuncAttributes f;
    return cudaFuncGetAttributes(&f, linear_split_kernel<CH>) == cudaSuccess && f.numRegs * (LS_THREADS / 32) >= 4 * 40 + 8 * 88 + 8 * 128;
  }();
  return enough;
}

// Bytes of working space for M rows of K numbers: three planes of bfloat16 and a scale per row.
extern "C" long long bn_linear_split_scratch(int M, int K) { return 6ll * M * ((K + 7) / 8 * 8) + 4ll * M; }

// x [M, K], w [N, K], out [M, ldo] float32, all 16-byte aligned with K a multiple of 4, 128 to 262,144; bias [N] or null; scratch as above.
extern "C" int bn_linear_split(const float* x, const float* w, const float* bias, float* out, int M, int N, int K, int ldo, void* scratch,
                               int* status, cudaStream_t stream) {
  if (M <= 0 || N <= 0) return BN_OK;
  if (!x || !w || !out || !scratch || !status || K < 4 * LS_BK || K % 4 || K > LS_MAX_K || ldo < N || ((uintptr_t)x | (uintptr_t)w | (uintptr_t)scratch) & 15 ||
      M > (1 << 28))
    return BN_ERR_BAD_ARG;
  const int pitch = (K + 7) / 8 * 8;
  __nv_bfloat16* planes = (__nv_bfloat16*)scratch;
  float* unscale = (float*)((unsigned char*)scratch + 6ll * M * pitch);
  LsArgs a = {};
  a.out = out; a.x = x; a.w = w; a.bias = bias; a.x_unscale = unscale;
  a.M = M; a.N = N; a.K = K; a.ldo = ldo; a.k_blocks = (K + LS_BK - 1) / LS_BK; a.status = status;
  a.n_tiles = (N + LS_BM - 1) / LS_BM;
  a.nt = ls_choose_nt(M, a.n_tiles, ls_sm_count());
  a.m_tiles = (M + a.nt - 1) / a.nt;
  if ((long long)a.n_tiles * a.m_tiles > 0x3fffffff) return BN_ERR_BAD_ARG;
  const int x_bytes = 3 * a.nt * LS_BK * 2, room = LS_SMEM_MAX - 1024 - LS_W_STAGES * LS_W_BYTES;
  a.x_stages = room / x_bytes < LS_X_STAGES_MAX ? room / x_bytes : LS_X_STAGES_MAX;
  CUtensorMap mw, mx;
  if (!ls_map(&mw, 3, w, N, K, 4ull * K, LS_BM) || !ls_map(&mx, 4, planes, 3ull * M, K, 2ull * pitch, a.nt)) return BN_ERR_BAD_ARG;
  BN_LAUNCH(linear_split_rows_kernel, M, 256, 0, stream, x, M, K, pitch, planes, unscale);
  const size_t smem = 1024 + LS_W_STAGES * LS_W_BYTES + (size_t)a.x_stages * x_bytes;
  const int tiles = a.n_tiles * a.m_tiles, grid = tiles < ls_sm_count() ? tiles : ls_sm_count();
#define LS_RUN(CH)                                                                                       \
  do {                                                                                                   \
    static BnGrant grant;                                                                                \
    if (!ls_registers<CH>()) return BN_ERR_BAD_ARG;                                                      \
    cudaError_t e = grant.ask((const void*)linear_split_kernel<CH>, smem, 1024);                         \
    if (e != cudaSuccess) return BN_ERR_LAUNCH + (int)e;                                                 \
    BN_LAUNCH((linear_split_kernel<CH>), grid, LS_THREADS, smem, stream, mw, mx, a);                     \
  } while (0)
  switch ((a.nt + 31) / 32) {
    case 1: LS_RUN(1); break;
    case 2: LS_RUN(2); break;
    case 3: LS_RUN(3); break;
    case 4: LS_RUN(4); break;
    case 5: LS_RUN(5); break;
    default: LS_RUN(6); break;
  }
  BN_CHECK_LAUNCH();
  return BN_OK;
}
