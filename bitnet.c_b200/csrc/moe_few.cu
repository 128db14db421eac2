// The expert products of a mixture for the few tokens of a decode step, in bfloat16: every chosen expert's matrices are read
// once for all the tokens that chose it.
//
//   bn_moe_few_gate_up  y[t * top + k] = act(W_gate[e] x, W_up[e] x), x = h[t] (times the weight, when it scales the input), e = ids[t][k]
//   bn_moe_few_down     out[t] = sum_k (weight) W_down[e] y[t * top + k] (+ what a shared expert gave), float32
//
// The products are bound by the experts' bytes.  Streaming them per (token, expert) item (moe.cu, which stays for float32, for
// sizes that are not whole 16-byte pieces, and where ops.moe_once_pays finds it faster) read an expert as often as tokens chose it:
// eight tokens with two of eight experts of
// 14336 + 7168 rows of 4096 took 393 us a layer (0.9 GB of different bytes, 135 us at the memory's rate).
// Here a warp multiplies 8 weight rows with up to 16 tokens at a time on the tensor cores (mma.sync m16n8k16, tokens as the 16
// rows): a lane's 16-byte piece of a weight row is at once its operand of two such instructions, because the order of the inner
// dimension is free as long as both operands take the same one.  Lanes copy the pieces of the weights and of the tokens' rows
// asynchronously into slots of their own in shared memory and read back only what they copied themselves, so a warp runs its
// stream of work, several stages ahead and across the ends of rows and experts, without any barrier.  (The same with the
// pieces in registers stood at 4.3 TB/s: loads return in order, so tokens' rows found in the L1 waited for the weights asked
// for ahead of them.)
//
// Which tokens chose an expert is worked out by every block for itself from the ids (a few hundred at most): a launch less.
#include "common.cuh"

#define MF_MAX_EXPERTS 1024
#define MF_MAX_ITEMS 128  // tokens times experts per token of one call; csrc/ops.py cuts its calls by the same numbers
// Row groups of 8 tokens that a warp multiplies with at a time (XR) and the stages of a warp's ring: a stage is, per lane, one
// 16-byte piece of each of the S weight streams and of each row group.  A block of 256 threads takes some 100 KB of shared memory,
// two of them an SM's, with some 130 KB of weights in flight with the fewest tokens.
#define MF_THREADS 256
#define MF_WARPS (MF_THREADS / 32)
// (S = 4: the rows of tokens serve twice as many weights, which is what counts with many of them)
__host__ __device__ constexpr int mf_stages(int S, int XR) { return 98 / (4 * (S + XR)); }
__host__ __device__ constexpr int mf_ring_bytes(int S, int XR) { return mf_stages(S, XR) * (S + XR) * 16 * MF_THREADS; }
// gate and up: the warps' parts of a unit's sums, [warp][8 XR tokens][S][8 rows], two of them in turn where that is small
__host__ __device__ constexpr int mf_part_floats(int S, int XR) { return MF_WARPS * 8 * XR * S * 8; }
__host__ __device__ constexpr int mf_part_turns(int S, int XR) { return S * XR <= 4 ? 2 : 1; }

struct MfArgs {
  const __nv_bfloat16* x;  // gate_up: h [tokens, width]; down: y [items, ff]
  const int* ids;
  const float* weights;
  int n_items, top, n_real;
  int K;                    // gate_up: width; down: ff
  int rows;                 // gate_up: ff; down: width
  const __nv_bfloat16 *w, *w_up;  // gate_up: the gate rows (or null) and the up rows; down: w and null
  size_t expert_stride;
  int scale_input;          // gate_up
  float limit, slope;
  int act;
  __nv_bfloat16* y;         // gate_up: [items, ff]
  int scale_output;         // down
  const void* add;
  int add_dtype;
  const float* add_scale;
  const __nv_bfloat16* h;   // down: the rows identity experts hand on
  float* out;
};

// 16 bytes into this lane's slot (zeros where there is nothing to copy: the address is then not read)
__device__ __forceinline__ void mf_copy_weights(unsigned dst, const __nv_bfloat16* src, bool live) {
  asm volatile("cp.async.cg.shared.global.L2::256B [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(live ? 16 : 0) : "memory");
}
__device__ __forceinline__ void mf_copy_row(unsigned dst, const __nv_bfloat16* src, bool live) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(live ? 16 : 0) : "memory");
}
__device__ __forceinline__ uint4 mf_slot(unsigned addr) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr) : "memory");
  return v;
}
// The sums of a group of 32 of the inner dimension, added to c: tokens' pieces x0 (rows g), x1 (rows g + 8), weights' piece w.  Each
// half is a product of its own from zero, and float32 additions do the rest: the tensor cores cut their sums off where an addition
// rounds, which along an inner dimension of 7,168 made the error against 64 bits 7 times that of float32 sums.
__device__ __forceinline__ void mf_mma(float* c, const uint4& x0, const uint4& x1, const uint4& w) {
  float d[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
               : "+f"(d[0][0]), "+f"(d[0][1]), "+f"(d[0][2]), "+f"(d[0][3]) : "r"(x0.x), "r"(x1.x), "r"(x0.y), "r"(x1.y), "r"(w.x), "r"(w.y));
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
               : "+f"(d[1][0]), "+f"(d[1][1]), "+f"(d[1][2]), "+f"(d[1][3]) : "r"(x0.z), "r"(x1.z), "r"(x0.w), "r"(x1.w), "r"(w.z), "r"(w.w));
#pragma unroll
  for (int i = 0; i < 4; ++i) c[i] += d[0][i] + d[1][i];
}
// part(0) + ... + part(MF_WARPS - 1), neighbours first
template <class Part>
__device__ __forceinline__ float mf_sum_of_warps(Part part) {
  float v[MF_WARPS];
#pragma unroll
  for (int w = 0; w < MF_WARPS; ++w) v[w] = part(w);
#pragma unroll
  for (int n = MF_WARPS / 2; n > 0; n >>= 1)
#pragma unroll
    for (int w = 0; w < n; ++w) v[w] = v[2 * w] + v[2 * w + 1];
  return v[0];
}
// Eight bfloat16 times a number, rounded to bfloat16 again (the expert's input as the path that sorts tokens stores it)
__device__ __forceinline__ uint4 mf_scaled(uint4 v, float s) {
  __nv_bfloat162* p = reinterpret_cast<__nv_bfloat162*>(&v);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 f = __bfloat1622float2(p[i]);
    p[i] = __floats2bfloat162_rn(f.x * s, f.y * s);
  }
  return v;
}

// The items of every expert, one behind another: list[off[e]] .. list[off[e + 1] - 1], and the experts that have any, in order.
// Shared memory: off [n_real + 1], cur [n_real], used [n_real], list [n_items].  Returns how many are used.
struct MfLists {
  int *off, *cur, *used, *list;
};
__device__ __forceinline__ MfLists mf_place_lists(int* s, const MfArgs& a) {
  MfLists l;
  l.off = s;
  l.cur = l.off + a.n_real + 1;
  l.used = l.cur + a.n_real;
  l.list = l.used + a.n_real;
  return l;
}
__device__ int mf_lists(const MfLists& l, const MfArgs& a) {
  __shared__ int s_used;
  const int tid = threadIdx.x, lane = tid & 31;
  for (int e = tid; e < a.n_real; e += blockDim.x) l.cur[e] = 0;
  const int mine = tid < a.n_items ? a.ids[tid] : -1;  // at most MF_MAX_ITEMS items, and no fewer threads
  __syncthreads();
  const bool real = mine >= 0 && mine < a.n_real;
  if (real) atomicAdd(&l.cur[mine], 1);
  __syncthreads();
  if (tid < 32) {
    const int per = (a.n_real + 31) / 32, e0 = min(lane * per, a.n_real), e1 = min(e0 + per, a.n_real);
    int items = 0, experts = 0;
    for (int e = e0; e < e1; ++e) {
      items += l.cur[e];
      experts += l.cur[e] > 0;
    }
    int upto = items, eupto = experts;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int u = __shfl_up_sync(0xffffffffu, upto, o), v = __shfl_up_sync(0xffffffffu, eupto, o);
      if (lane >= o) { upto += u; eupto += v; }
    }
    int at = upto - items, eat = eupto - experts;
    for (int e = e0; e < e1; ++e) {
      const int n = l.cur[e];
      l.off[e] = at;
      l.cur[e] = at;
      at += n;
      if (n) l.used[eat++] = e;
    }
    if (lane == 31) {
      l.off[a.n_real] = upto;
      s_used = eupto;
    }
  }
  __syncthreads();
  if (real) l.list[atomicAdd(&l.cur[mine], 1)] = tid;
  __syncthreads();
  return s_used;
}

// A warp's place in its stream of work: 8 weight rows of an expert (S matrices) times the rows of up to 8 XR of its tokens, 32
// numbers of the inner dimension at a time.  `u` counts the stream's units, `m0` the expert's tokens, `k` the inner dimension.
#define MF_NO_ROW 0xffffffffu
template <int S, int XR>
struct MfCursor {
  int u, m0, n, first, k;
  const __nv_bfloat16* w[S];  // this lane's weight rows
  unsigned x[XR];             // where this lane's rows begin in x
};

// Runs a warp's stream.  `open(cursor)` fills in a unit's expert, its tokens and the lane's weight rows from cursor.u (false: no
// such unit); `row(item)` the row of x that an item takes; `next(u)` the unit after u; `finish(cursor, acc)` takes the sums.  A warp
// whose share k0 .. k1 is empty takes one piece of nothing per sum.  AHEAD: the first stages' weights are asked for before the wait for
// the kernel before this one, the rows behind it.
template <int S, int XR, bool SCALED, bool AHEAD, class Open, class Row, class Next, class Finish>
__device__ __forceinline__ void mf_stream(const MfArgs& a, const MfLists& l, unsigned ring, int u0, int k0, int k1, Open open, Row row, Next next,
                                          Finish finish) {
  constexpr int D = mf_stages(S, XR), MT = (XR + 1) / 2;
  const int lane = threadIdx.x & 31, g = lane >> 2, quad = lane & 3;
  const unsigned slot_bytes = blockDim.x * 16, stage_bytes = slot_bytes * (S + XR);
  ring += threadIdx.x * 16;
  MfCursor<S, XR> f, c;  // what is asked for; what is multiplied
  auto rows = [&](MfCursor<S, XR>& q) {
#pragma unroll
    for (int i = 0; i < XR; ++i) {
      const int r = q.m0 + i * 8 + g;
      q.x[i] = r < q.n ? (unsigned)row(l.list[q.first + r]) * (unsigned)a.K : MF_NO_ROW;
    }
  };
  auto step = [&](MfCursor<S, XR>& q, bool& live, bool with_rows) {  // to the next piece; true at the end of a sum
    q.k += 32;
    if (q.k < k1) return false;
    q.k = k0;
    q.m0 += 8 * XR;
    if (q.m0 >= q.n) {
      q.u = next(q.u);
      q.m0 = 0;
      live = open(q);
    }
    if (live && with_rows) rows(q);
    return true;
  };
  bool more = true, live = true;
  f.u = c.u = u0;
  f.m0 = c.m0 = 0;
  f.k = c.k = k0;
  more = live = open(f);
  if (!live) return;
  if (!AHEAD) rows(f);
  open(c);
  float acc[MT][S][4], xs[XR];
  auto clear = [&]() {
#pragma unroll
    for (int m = 0; m < MT; ++m)
#pragma unroll
      for (int s = 0; s < S; ++s)
#pragma unroll
        for (int i = 0; i < 4; ++i) acc[m][s][i] = 0.f;
    if (SCALED) {
#pragma unroll
      for (int i = 0; i < XR; ++i) {
        const int r = c.m0 + i * 8 + g;
        xs[i] = r < c.n ? a.weights[l.list[c.first + r]] : 0.f;
      }
    }
  };
  auto fetch = [&](int stage, bool weights, bool x) {
    if (more) {
      const int at = f.k + quad * 8;
      const unsigned dst = ring + stage * stage_bytes;
      if (weights) {
#pragma unroll
        for (int s = 0; s < S; ++s) mf_copy_weights(dst + s * slot_bytes, f.w[s] + at, at < k1);
      }
      if (x) {
#pragma unroll
        for (int i = 0; i < XR; ++i) {
          const bool have = f.x[i] != MF_NO_ROW && at < k1;
          mf_copy_row(dst + (S + i) * slot_bytes, a.x + (have ? f.x[i] + at : 0u), have);
        }
      }
      step(f, more, x);
    }
    if (x) asm volatile("cp.async.commit_group;" ::: "memory");
  };
  int stage = 0;
  if (AHEAD) {
#pragma unroll 1
    for (; stage < D - 1; ++stage) fetch(stage, true, false);
    pdl_wait();
    f = c;
    more = true;
    rows(f);
  }
#pragma unroll 1
  for (stage = 0; stage < D - 1; ++stage) fetch(stage, !AHEAD, true);
  clear();
  int at = 0;
#pragma unroll 1
  while (live) {
    asm volatile("cp.async.wait_group %0;" ::"n"(D - 2) : "memory");  // the oldest stage has landed
    fetch(stage, true, true);  // into the stage that was read one turn ago
    stage = stage + 1 == D ? 0 : stage + 1;
    const unsigned src = ring + at * stage_bytes;
    at = at + 1 == D ? 0 : at + 1;
    uint4 w[S];
#pragma unroll
    for (int s = 0; s < S; ++s) w[s] = mf_slot(src + s * slot_bytes);
#pragma unroll
    for (int m = 0; m < MT; ++m) {
      uint4 x0 = mf_slot(src + (S + 2 * m) * slot_bytes), x1 = make_uint4(0u, 0u, 0u, 0u);
      if (2 * m + 1 < XR) x1 = mf_slot(src + (S + 2 * m + 1) * slot_bytes);
      if (SCALED) {
        x0 = mf_scaled(x0, xs[2 * m]);
        if (2 * m + 1 < XR) x1 = mf_scaled(x1, xs[2 * m + 1]);
      }
#pragma unroll
      for (int s = 0; s < S; ++s) mf_mma(acc[m][s], x0, x1, w[s]);
    }
    const MfCursor<S, XR> done = c;
    if (step(c, live, false)) {
      finish(done, acc);
      if (live) clear();
    }
  }
}

// A unit of work: 8 rows (of both matrices, where there is a gate) of one used expert.  A block takes one at a time, its warps share
// out the inner dimension (the same way whatever the batch) and their parts are added in shared memory: one warp per unit left a
// last wave nearly empty (three experts of 896 units on 2368 warps) and SMs without work (eight experts of 128 units).
template <int G, int R, int XR, bool SCALED>  // G matrices, R times 8 rows of each
__global__ void __launch_bounds__(MF_THREADS, 2) moe_few_gate_up_kernel(MfArgs a) {
  constexpr int S = G * R, TURNS = mf_part_turns(S, XR);
  pdl_wait();
  pdl_launch_dependents();  // not before: what follows relies on the ids being there
  extern __shared__ __align__(16) unsigned char mf_smem[];
  const unsigned ring = (unsigned)__cvta_generic_to_shared(mf_smem);
  float* parts = (float*)(mf_smem + mf_ring_bytes(S, XR));
  const MfLists l = mf_place_lists((int*)(parts + TURNS * mf_part_floats(S, XR)), a);
  const int used = mf_lists(l, a);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, quad = lane & 3;
  const int tiles = a.rows / (8 * R), units = used * tiles;
  const int pieces = (a.K + 31) / 32, per = (pieces + MF_WARPS - 1) / MF_WARPS;
  const int k0 = warp * per * 32, k1 = min(a.K, k0 + per * 32);
  int turn = 0;
  mf_stream<S, XR, SCALED, false>(
      a, l, ring, blockIdx.x, k0, k1,
      [&](MfCursor<S, XR>& q) {
        if (q.u >= units) return false;
        const int e = l.used[q.u / tiles];
        q.first = l.off[e];
        q.n = l.off[e + 1] - q.first;
        const size_t at = (size_t)e * a.expert_stride + (size_t)((q.u % tiles) * 8 * R + g) * a.K;
#pragma unroll
        for (int i = 0; i < R; ++i) {
          q.w[i] = (G == 2 ? a.w : a.w_up) + at + (size_t)i * 8 * a.K;
          if (G == 2) q.w[S - R + i] = a.w_up + at + (size_t)i * 8 * a.K;
        }
        return true;
      },
      [&](int item) { return item / a.top; }, [&](int u) { return u + (int)gridDim.x; },
      [&](const MfCursor<S, XR>& q, float(*acc)[S][4]) {
        // with two, who still reads the other one has not passed the barrier below, and nobody passes it again before that
        float* part = parts + turn * mf_part_floats(S, XR);
        if (TURNS == 2) turn ^= 1;
        else __syncthreads();
#pragma unroll
        for (int i = 0; i < XR; ++i)
#pragma unroll
          for (int s = 0; s < S; ++s)
            *reinterpret_cast<float2*>(part + ((warp * 8 * XR + i * 8 + g) * S + s) * 8 + quad * 2) =
                make_float2(acc[i / 2][s][2 * (i & 1)], acc[i / 2][s][2 * (i & 1) + 1]);
        __syncthreads();
        const int n = min(q.n - q.m0, 8 * XR);
        for (int o = threadIdx.x; o < n * 8 * R; o += MF_THREADS) {
          const int r = o / (8 * R), j = o % (8 * R);
          float sum[G];
#pragma unroll
          for (int m = 0; m < G; ++m) {
            sum[m] = mf_sum_of_warps([&](int w) { return part[((w * 8 * XR + r) * S + m * R) * 8 + j]; });
          }
          // the products' results pass through bfloat16, as they do on the sorted path
          const float up = to_f32<__nv_bfloat16>(from_f32<__nv_bfloat16>(sum[G - 1]));
          float v;
          if (G == 1) {
            v = relu_squared(up);
          } else {
            const float gate = to_f32<__nv_bfloat16>(from_f32<__nv_bfloat16>(sum[0]));
            if (a.act >= 0) {
              v = glu_activation(gate, a.act) * up;
            } else {
              const float gl = fminf(gate, a.limit);
              v = gl / (1.0f + expf(-a.slope * gl)) * (fminf(fmaxf(up, -a.limit), a.limit) + 1.0f);
            }
          }
          a.y[(size_t)l.list[q.first + q.m0 + r] * a.rows + (q.u % tiles) * 8 * R + j] = from_f32<__nv_bfloat16>(v);
        }
      });
}

// A block: 8 R rows of every used expert's matrix; its warps share out the inner dimension (the same way whatever the batch) and
// leave their parts of every item's result in shared memory, [warp][item][8 R].  Then each token's items are added in their order.
// Launched behind the kernel above, which lets it begin only when the ids are there: lists and the first weights need no wait.
template <int R, int XR>
__global__ void __launch_bounds__(MF_THREADS, 2) moe_few_down_kernel(MfArgs a) {
  pdl_launch_dependents();
  extern __shared__ __align__(16) unsigned char mf_smem[];
  const unsigned ring = (unsigned)__cvta_generic_to_shared(mf_smem);
  float* parts = (float*)(mf_smem + mf_ring_bytes(R, XR));
  const MfLists l = mf_place_lists((int*)(parts + MF_WARPS * a.n_items * 8 * R), a);
  const int used = mf_lists(l, a);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, quad = lane & 3;
  const int c0 = blockIdx.x * 8 * R;
  const int pieces = (a.K + 31) / 32, per = (pieces + MF_WARPS - 1) / MF_WARPS;
  const int k0 = warp * per * 32, k1 = min(a.K, k0 + per * 32);
  float* part = parts + (size_t)warp * a.n_items * 8 * R;
  mf_stream<R, XR, false, true>(
      a, l, ring, 0, k0, k1,
      [&](MfCursor<R, XR>& q) {
        if (q.u >= used) return false;
        const int e = l.used[q.u];
        q.first = l.off[e];
        q.n = l.off[e + 1] - q.first;
#pragma unroll
        for (int i = 0; i < R; ++i) q.w[i] = a.w + (size_t)e * a.expert_stride + (size_t)(c0 + i * 8 + g) * a.K;
        return true;
      },
      [&](int item) { return item; }, [&](int u) { return u + 1; },
      [&](const MfCursor<R, XR>& q, float(*acc)[R][4]) {
#pragma unroll
        for (int i = 0; i < XR; ++i) {
          const int r = q.m0 + i * 8 + g;
          if (r < q.n)
#pragma unroll
            for (int s = 0; s < R; ++s)
              *reinterpret_cast<float2*>(part + ((size_t)l.list[q.first + r] * R + s) * 8 + quad * 2) =
                  make_float2(acc[i / 2][s][2 * (i & 1)], acc[i / 2][s][2 * (i & 1) + 1]);
        }
      });
  pdl_wait();  // (a block without a stream has not waited)
  __syncthreads();
  const int n_tokens = a.n_items / a.top;
  for (int o = threadIdx.x; o < n_tokens * 8 * R; o += MF_THREADS) {
    const int t = o / (8 * R), r = o % (8 * R);
    float total = 0.f;
    for (int k = 0; k < a.top; ++k) {
      const int item = t * a.top + k, e = a.ids[item];
      float d = 0.f;
      if (e >= a.n_real) {
        d = to_f32<__nv_bfloat16>(a.h[(size_t)t * a.rows + c0 + r]);
      } else if (e >= 0) {
        d = mf_sum_of_warps([&](int q) { return parts[((size_t)q * a.n_items + item) * 8 * R + r]; });
      }
      total += d * (a.scale_output ? a.weights[item] : 1.0f);
    }
    if (a.add) total += load_as_f32(a.add, a.add_dtype, (size_t)t * a.rows + c0 + r) * (a.add_scale ? a.add_scale[t] : 1.0f);
    a.out[(size_t)t * a.rows + c0 + r] = total;
  }
}

static int mf_sm_count() {
  static int n = 0;
  if (!n) {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0)
      n = 148;
  }
  return n;
}
static size_t mf_list_bytes(const MfArgs& a) { return (size_t)(3 * a.n_real + 1 + a.n_items) * sizeof(int); }

#define MF_SMEM_MAX (180 * 1024)
// out [n_tokens, width] float32 from h [n_tokens, width], ids and weights [n_tokens, top]: both products of every chosen expert, with
// y [n_tokens * top, ff] between them.  w_gate (null: the square of relu(up)) and w_up: row j of expert e lies at e * expert_stride +
// j * width; w_down [experts, width, ff].  act < 0: the clamped unit with `limit` and `slope`; else act(gate) * up.  The weights
// multiply the experts' input (scale_input) or output.  add [n_tokens, width] of add_dtype (or null), its rows times add_scale
// [n_tokens] (or null).  Ids from n_real on are identity experts, whose output is the token's row of h.  width and ff are multiples of
// 8, matrices and rows of bfloat16 16-byte aligned, n_tokens * top at most MF_MAX_ITEMS.
extern "C" int bn_moe_few(const void* h, int n_tokens, int width, const int* ids, const float* weights, int scale_input, const void* w_gate,
                          const void* w_up, long long expert_stride, int ff, int top, float limit, float slope, int act, int n_real, void* y,
                          const void* w_down, const void* add, int add_dtype, const float* add_scale, float* out, cudaStream_t stream) {
  if (n_tokens <= 0) return BN_OK;
  if (!h || !ids || !weights || !w_up || !w_down || !y || !out || top <= 0 || top > MF_MAX_ITEMS || n_tokens > MF_MAX_ITEMS / top ||
      n_real <= 0 || n_real > MF_MAX_EXPERTS || width <= 0 || width % 8 || ff <= 0 || ff % 8 || expert_stride % 8 || width > (1 << 24) ||
      ff > (1 << 24) ||  // 128 rows of x in 32-bit offsets
      (((uintptr_t)h | (uintptr_t)w_gate | (uintptr_t)w_up | (uintptr_t)w_down | (uintptr_t)y) & 15))
    return BN_ERR_BAD_ARG;
  MfArgs a = {};
  a.x = (const __nv_bfloat16*)h; a.ids = ids; a.weights = weights; a.n_items = n_tokens * top; a.top = top; a.n_real = n_real;
  a.K = width; a.rows = ff; a.w = (const __nv_bfloat16*)w_gate; a.w_up = (const __nv_bfloat16*)w_up; a.expert_stride = (size_t)expert_stride;
  a.scale_input = scale_input; a.limit = limit; a.slope = slope; a.act = act; a.y = (__nv_bfloat16*)y;
  // Row groups by the average number of items per expert (one with more passes its weights again, from the L2), and with
  // two twice the rows: at 64 tokens with 2 of 8 experts the tokens' rows were half of what was copied.
  const int xr = a.n_items <= 5 * n_real || n_tokens <= 8 ? 1 : a.n_items <= 16 * n_real || n_tokens <= 16 ? 2 : 4;
  const int twice = xr == 2 && ff % 16 == 0 ? 2 : 1;
  const long long units = (long long)(a.n_items < n_real ? a.n_items : n_real) * (ff / (8 * twice)), most = 2LL * mf_sm_count();
  const unsigned grid = (unsigned)(units < most ? units : most);
#define MF_UP(G, R, XR, SCALED)                                                                                                 \
  do {                                                                                                                          \
    const size_t smem = mf_ring_bytes(G * R, XR) + mf_part_turns(G * R, XR) * mf_part_floats(G * R, XR) * sizeof(float) + mf_list_bytes(a); \
    static BnGrant grant;                                                                                                       \
    if (smem > MF_SMEM_MAX) return BN_ERR_BAD_ARG;                                                                              \
    cudaError_t e = grant.ask((const void*)moe_few_gate_up_kernel<G, R, XR, SCALED>, smem, 1024);                               \
    if (e != cudaSuccess) return BN_ERR_LAUNCH + (int)e;                                                                        \
    BN_LAUNCH((moe_few_gate_up_kernel<G, R, XR, SCALED>), grid, MF_THREADS, smem, stream, a);                                   \
  } while (0)
#define MF_UP_ROWS(G, SCALED)                              \
  do {                                                     \
    if (xr == 1) MF_UP(G, 1, 1, SCALED);                   \
    else if (xr == 2 && twice == 2) MF_UP(G, 2, 2, SCALED); \
    else if (xr == 2) MF_UP(G, 1, 2, SCALED);              \
    else MF_UP(G, 1, 4, SCALED);                           \
  } while (0)
  if (w_gate && scale_input) MF_UP_ROWS(2, true);
  else if (w_gate) MF_UP_ROWS(2, false);
  else if (scale_input) MF_UP_ROWS(1, true);
  else MF_UP_ROWS(1, false);
  a.x = (const __nv_bfloat16*)y;
  a.K = ff; a.rows = width; a.w = (const __nv_bfloat16*)w_down; a.w_up = nullptr; a.expert_stride = (size_t)width * ff;
  a.scale_output = !scale_input; a.add = add; a.add_dtype = add_dtype; a.add_scale = add_scale; a.h = (const __nv_bfloat16*)h; a.out = out;
  // 16 rows per block where that leaves a block per SM: 512 blocks of 8 rows (width 4096) took a second, mostly empty, wave
  const int wide = width % 16 == 0 && width / 16 >= mf_sm_count() && a.n_items * 16 * MF_WARPS * (int)sizeof(float) <= 64 * 1024;
#define MF_DOWN(R, XR)                                                                                                          \
  do {                                                                                                                          \
    const size_t smem = mf_ring_bytes(R, XR) + (size_t)MF_WARPS * a.n_items * 8 * R * sizeof(float) + mf_list_bytes(a);         \
    static BnGrant grant;                                                                                                       \
    if (smem > MF_SMEM_MAX) return BN_ERR_BAD_ARG;                                                                              \
    cudaError_t e = grant.ask((const void*)moe_few_down_kernel<R, XR>, smem, 1024);                                             \
    if (e != cudaSuccess) return BN_ERR_LAUNCH + (int)e;                                                                        \
    BN_LAUNCH((moe_few_down_kernel<R, XR>), (unsigned)(width / (8 * R)), MF_THREADS, smem, stream, a);                          \
  } while (0)
  if (xr == 1 && wide) MF_DOWN(2, 1);
  else if (xr == 1) MF_DOWN(1, 1);
  else if (xr == 2 && wide) MF_DOWN(2, 2);
  else if (xr == 2) MF_DOWN(1, 2);
  else if (wide) MF_DOWN(2, 4);
  else MF_DOWN(1, 4);
  BN_CHECK_LAUNCH();
  return BN_OK;
}

// ---- the same products with the sums of moe.cu ------------------------------------------------------------------------------------
//
//   bn_moe_few_in_order  out[t] as bn_moe_gate_up_ex and bn_moe_down of moe.cu give it, bit for bit
//
// For designs whose next token would fall to another order of summation (MoeSpec.read_once = False): a lane takes pieces of eight
// numbers, 256 apart, multiplies and adds them one after another in float32, and the 32 lanes' sums meet in a butterfly.  The tensor
// cores have no such order; the float32 units have time for it as long as an expert has few tokens.
//
// One block per SM.  A block keeps the rows of x of the tokens that chose an expert in shared memory (as many as fit: `cap`; an expert
// with more is passed over again); it takes a run of all experts' rows, whose part of each expert its warps share in half units, and a warp
// streams 8 rows at a time (4 of each matrix, where there are two; half of that where no more are left) through slots of its lanes' own,
// copied D - 1 stages ahead.  Runs are cut at any row, and a row counts MR_ROW_COST + its tokens: with equal runs the blocks of the expert
// that most tokens chose were the last by far.  (With a run for every warp of its own, cut from all rows alike, half of a block's warps
// waited for the others wherever a block's run went from one expert to the next: 8 experts of 4096 x 7168, 8 tokens 280 -> 185 us, 16 tokens
// 398 -> 263, 64 tokens 1270 -> 730; 64 of 2048 x 1408, 16 tokens 124.)
// A piece of x serves eight rows, two of them with each instruction (fma.rn.f32x2: two float32 multiply-adds, each rounded as one alone).
#define MR_WARPS 8
#define MR_THREADS (32 * MR_WARPS)
#define MR_S 8       // rows of weights a warp multiplies with at a time
#define MR_TOKENS 8  // tokens a pass takes at most
#define MR_ROW_COST 4
#define MR_SMEM_MAX (226 * 1024)
__host__ __device__ constexpr int mr_ring_bytes(int D) { return MR_WARPS * D * MR_S * 512; }

struct MrArgs {
  MfArgs m;
  int cap;   // tokens of an expert that one pass takes
  float* d;  // the last product (else null): [items, rows] every item's product
};

__device__ __forceinline__ float mr_low(unsigned v) { return __uint_as_float(v << 16); }
__device__ __forceinline__ float mr_high(unsigned v) { return __uint_as_float(v & 0xffff0000u); }
__device__ __forceinline__ unsigned long long mr_pair(float a, float b) {
  unsigned long long v;
  asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(a), "f"(b));
  return v;
}
// The sums over the warp's lanes of v[0 .. C - 1], each by the additions of warp_sum: lane l meets l ^ O.  Where there is an even number of
// them left, a lane goes on with half: v[0 ..] are then the numbers from mr_fold_first(C, lane) on.
template <int C, int O>
__device__ __forceinline__ void mr_fold(float* v, int lane) {
  if constexpr (O > 0 && C % 2 == 0) {
    const bool upper = lane & O;
#pragma unroll
    for (int i = 0; i < C / 2; ++i) {
      const float send = upper ? v[i] : v[i + C / 2], keep = upper ? v[i + C / 2] : v[i];
      v[i] = keep + __shfl_xor_sync(0xffffffffu, send, O);
    }
    mr_fold<C / 2, O / 2>(v, lane);
  } else if constexpr (O > 0) {
#pragma unroll
    for (int i = 0; i < C; ++i) v[i] += __shfl_xor_sync(0xffffffffu, v[i], O);
    mr_fold<C, O / 2>(v, lane);
  }
}
__host__ __device__ constexpr int mr_fold_left(int c) {  // how many numbers a lane ends with
  for (int o = 16; o > 0; o >>= 1)
    if (c % 2 == 0) c /= 2;
  return c;
}
__device__ __forceinline__ int mr_fold_first(int c, int lane) {
  int first = 0;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
    if (c % 2 == 0) {
      c /= 2;
      if (lane & o) first += c;
    }
  return first;
}

// The passes over experts: seg_expert[s] and the first of its tokens seg_m0[s]; returns how many there are (at most n_items).
// seg_cost[s]: what a row of every pass before s costs, seg_cost[passes] a row of all.
__device__ int mr_passes(const MfArgs& a, const MfLists& l, int used, int cap, int* seg_expert, int* seg_m0, int* seg_cost) {
  __shared__ int s_passes;
  // The items of an expert in their order: every block has to cut them into the same passes (mf_lists leaves them as they come).
  int e = -1, place = 0;
  if (threadIdx.x < a.n_items) {
    e = a.ids[threadIdx.x];
    if (e < 0 || e >= a.n_real) e = -1;
    else for (int i = l.off[e]; i < l.off[e + 1]; ++i) place += l.list[i] < (int)threadIdx.x;
  }
  __syncthreads();
  if (e >= 0) l.list[l.off[e] + place] = threadIdx.x;
  constexpr int PER = MF_MAX_ITEMS / 32;  // used experts, and passes, a lane takes
  if (threadIdx.x < 32) {
    const int lane = threadIdx.x;
    int n[PER], mine = 0;
#pragma unroll
    for (int i = 0; i < PER; ++i) {
      const int u = lane * PER + i;
      n[i] = u < used ? (l.off[l.used[u] + 1] - l.off[l.used[u]] + cap - 1) / cap : 0;
      mine += n[i];
    }
    int upto = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, upto, o);
      if (lane >= o) upto += v;
    }
    int at = upto - mine;
#pragma unroll
    for (int i = 0; i < PER; ++i)
      for (int p = 0; p < n[i]; ++p) {
        seg_expert[at] = l.used[lane * PER + i];
        seg_m0[at++] = p * cap;
      }
    if (lane == 31) s_passes = upto;
    __syncwarp();
    const int passes = __shfl_sync(0xffffffffu, upto, 31);
    int cost[PER], sum = 0;
#pragma unroll
    for (int i = 0; i < PER; ++i) {
      const int s = lane * PER + i;
      cost[i] = 0;
      if (s < passes) {
        const int x = seg_expert[s];
        cost[i] = MR_ROW_COST + min(cap, l.off[x + 1] - l.off[x] - seg_m0[s]);
      }
      sum += cost[i];
    }
    upto = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, upto, o);
      if (lane >= o) upto += v;
    }
    at = upto - sum;
#pragma unroll
    for (int i = 0; i < PER; ++i) {
      const int s = lane * PER + i;
      if (s <= passes) seg_cost[s] = at;
      at += cost[i];
    }
    if (lane == 31 && passes == MF_MAX_ITEMS) seg_cost[passes] = at;
  }
  __syncthreads();
  return s_passes;
}

// What a warp streams in one pass: rows 0 .. n_rows - 1 behind w (and w_up), pieces of 256 numbers.
struct MrStream {
  const __nv_bfloat16 *w, *w_up;  // this lane's first number of its first row
  int n_rows, pieces, K, in_row;  // in_row: numbers of a row from this lane's first on
  unsigned ring;                  // this lane's first slot
  int fj, fk, f_stage, stage;     // asked for: rows from fj on, piece fk, into f_stage; read next: stage
};
// Rows of each matrix in the unit that begins with `left` rows left
template <int G>
__device__ __forceinline__ int mr_unit(int left) { return left > MR_S / G / 2 ? MR_S / G : MR_S / G / 2; }

template <int G, int D>
__device__ __forceinline__ void mr_fetch(MrStream& q) {
  const int left = q.n_rows - q.fj;
  if (left > 0) {
    const int unit = mr_unit<G>(left);
    if (q.fk * 256 < q.in_row) {
      const size_t at = (size_t)q.fj * q.K + q.fk * 256;
      const unsigned dst = q.ring + q.f_stage * (MR_S * 512);
#pragma unroll
      for (int r = 0; r < MR_S / G; ++r)
        if (r < left) {  // (never more than a unit: what is left of a smaller one is at most its size)
          mf_copy_weights(dst + r * 512, q.w + at + (size_t)r * q.K, true);
          if (G == 2) mf_copy_weights(dst + (unit + r) * 512, q.w_up + at + (size_t)r * q.K, true);
        }
    }
    if (++q.fk == q.pieces) {
      q.fk = 0;
      q.fj += unit;
    }
  }
  asm volatile("cp.async.commit_group;" ::: "memory");
  q.f_stage = q.f_stage + 1 == D ? 0 : q.f_stage + 1;
}

// One unit: R rows (of all matrices together) times N tokens, whose rows begin at x; the sums go to out [N][R].
template <int G, int D, int N, int R>
__device__ __forceinline__ void mr_rows(MrStream& q, const __nv_bfloat16* x, float* out, int lane) {
  unsigned long long acc[N][R / 2];
#pragma unroll
  for (int t = 0; t < N; ++t)
#pragma unroll
    for (int r = 0; r < R / 2; ++r) acc[t][r] = 0ull;
#pragma unroll 1
  for (int k = 0; k < q.pieces; ++k) {
    asm volatile("cp.async.wait_group %0;" ::"n"(D - 2) : "memory");  // the oldest stage has landed
    unsigned w[R][4], xs[N][4];
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const uint4 v = mf_slot(q.ring + (q.stage * MR_S + r) * 512);
      w[r][0] = v.x; w[r][1] = v.y; w[r][2] = v.z; w[r][3] = v.w;
    }
    q.stage = q.stage + 1 == D ? 0 : q.stage + 1;
    const bool live = k * 256 < q.in_row;
#pragma unroll
    for (int t = 0; t < N; ++t) {
      uint4 v = make_uint4(0u, 0u, 0u, 0u);
      if (live) v = *reinterpret_cast<const uint4*>(x + (size_t)t * q.K + k * 256);
      xs[t][0] = v.x; xs[t][1] = v.y; xs[t][2] = v.z; xs[t][3] = v.w;
    }
    mr_fetch<G, D>(q);  // into the stage that was read one turn ago
    if (live) {
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        unsigned long long wp[R / 2];
#pragma unroll
        for (int r = 0; r < R / 2; ++r)
          wp[r] = i & 1 ? mr_pair(mr_high(w[2 * r][i / 2]), mr_high(w[2 * r + 1][i / 2])) : mr_pair(mr_low(w[2 * r][i / 2]), mr_low(w[2 * r + 1][i / 2]));
#pragma unroll
        for (int t = 0; t < N; ++t) {
          const float v = i & 1 ? mr_high(xs[t][i / 2]) : mr_low(xs[t][i / 2]);
          const unsigned long long xx = mr_pair(v, v);
#pragma unroll
          for (int r = 0; r < R / 2; ++r) asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc[t][r]) : "l"(xx), "l"(wp[r]));
        }
      }
    }
  }
  float v[N * R];
#pragma unroll
  for (int t = 0; t < N; ++t)
#pragma unroll
    for (int r = 0; r < R / 2; ++r) asm("mov.b64 {%0, %1}, %2;" : "=f"(v[t * R + 2 * r]), "=f"(v[t * R + 2 * r + 1]) : "l"(acc[t][r]));
  mr_fold<N * R, 16>(v, lane);
  const int first = mr_fold_first(N * R, lane);
#pragma unroll
  for (int i = 0; i < mr_fold_left(N * R); ++i) out[first + i] = v[i];
}

// G matrices: 2, gate and up; 1, up alone, or the last product's
template <int G, int D>
__global__ void __launch_bounds__(MR_THREADS, 1) moe_in_order_kernel(MrArgs p) {
  const MfArgs& a = p.m;
  const bool down = p.d != nullptr;
  if (!down) pdl_wait();
  pdl_launch_dependents();  // (gate and up: not before, the last product's blocks rely on the ids being there)
  extern __shared__ __align__(16) unsigned char mr_smem[];
  __shared__ float s_sums[MR_WARPS][MR_TOKENS * MR_S];
  __nv_bfloat16* xs = (__nv_bfloat16*)(mr_smem + mr_ring_bytes(D));  // [cap][K]
  const MfLists l = mf_place_lists((int*)(xs + (size_t)p.cap * a.K), a);
  int *seg_expert = l.list + a.n_items, *seg_m0 = seg_expert + a.n_items, *seg_cost = seg_m0 + a.n_items;  // (the last: one number more)
  const int used = mf_lists(l, a);
  const int passes = mr_passes(a, l, used, p.cap, seg_expert, seg_m0, seg_cost);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  // The run of block b: rows whose cost lies in [b, b + 1) of gridDim.x equal shares.  cut(b): a pass and a row in it.
  const long long total = (long long)seg_cost[passes] * a.rows;
  auto cut = [&](int b, int& row) {
    const long long at = total * b / gridDim.x;
    int seg = 0;
    while (seg < passes && (long long)seg_cost[seg + 1] * a.rows <= at) ++seg;
    row = seg < passes ? (int)((at - (long long)seg_cost[seg] * a.rows) / (seg_cost[seg + 1] - seg_cost[seg])) : 0;
    return seg;
  };
  int row0, row1;
  const int seg0 = cut(blockIdx.x, row0), seg1 = cut(blockIdx.x + 1, row1);  // from row0 of pass seg0 to before row1 of pass seg1
  MrStream q;
  q.K = a.K;
  q.pieces = (a.K + 255) / 256;
  q.in_row = a.K - lane * 8;
  q.ring = (unsigned)__cvta_generic_to_shared(mr_smem) + warp * (D * MR_S * 512) + lane * 16;
  bool waited = !down;

  for (int seg = seg0; seg < passes && seg <= seg1; ++seg) {
    // the warps share the block's rows of this pass, in half units
    const int b0 = seg == seg0 ? row0 : 0, b1 = seg < seg1 ? a.rows : row1, halves = (b1 - b0 + MR_S / G / 2 - 1) / (MR_S / G / 2);
    if (halves <= 0) continue;
    const int j0 = b0 + halves * warp / MR_WARPS * (MR_S / G / 2), j1 = min(b1, b0 + halves * (warp + 1) / MR_WARPS * (MR_S / G / 2));
    const int e = seg_expert[seg], first = l.off[e] + seg_m0[seg];
    const int n = min(p.cap, l.off[e + 1] - first);
    const size_t at = (size_t)e * a.expert_stride + (size_t)j0 * a.K + lane * 8;
    q.w = (G == 2 ? a.w : a.w_up) + at;
    q.w_up = a.w_up + at;
    q.n_rows = j1 > j0 ? j1 - j0 : 0;
    q.fj = q.fk = q.f_stage = q.stage = 0;
#pragma unroll 1
    for (int i = 0; i < D - 1; ++i) mr_fetch<G, D>(q);
    if (!waited) {
      pdl_wait();
      waited = true;
    }
    __syncthreads();  // nobody reads the rows of the pass before any more
    for (int t = 0; t < n; ++t) {  // the rows of x
      const int item = l.list[first + t];
      const __nv_bfloat16* src = a.x + (size_t)(down ? item : item / a.top) * a.K;
      __nv_bfloat16* dst = xs + (size_t)t * a.K;
      if (!down && a.scale_input) {
        const float s = a.weights[item];
#pragma unroll 4
        for (int c = tid * 8; c < a.K; c += MR_THREADS * 8) *reinterpret_cast<uint4*>(dst + c) = mf_scaled(*reinterpret_cast<const uint4*>(src + c), s);
      } else {
        for (int c = tid * 8; c < a.K; c += MR_THREADS * 8) mf_copy_weights((unsigned)__cvta_generic_to_shared(dst + c), src + c, true);
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    const __nv_bfloat16* x = xs + lane * 8;
    float* sums = s_sums[warp];
    for (int j = 0; j < q.n_rows;) {
      const int unit = mr_unit<G>(q.n_rows - j);
#define MR_CASE(N)                                                             \
  case N:                                                                      \
    if (unit == MR_S / G) mr_rows<G, D, N, MR_S>(q, x, sums, lane);            \
    else mr_rows<G, D, N, MR_S / 2>(q, x, sums, lane);                         \
    break
      switch (n) {
        MR_CASE(1); MR_CASE(2); MR_CASE(3); MR_CASE(4); MR_CASE(5); MR_CASE(6); MR_CASE(7); MR_CASE(8);
      }
#undef MR_CASE
      __syncwarp();
      const int rows = min(unit, q.n_rows - j);
      for (int o = lane; o < n * unit; o += 32) {
        const int t = o / unit, r = o - t * unit;
        if (r >= rows) continue;
        const int item = l.list[first + t];
        const size_t to = (size_t)item * a.rows + j0 + j + r;
        const float last = sums[t * unit * G + (G - 1) * unit + r];
        if (down) {
          p.d[to] = last;
          continue;
        }
        // the products' results pass through bfloat16, as they do on the sorted path
        const float up = to_f32<__nv_bfloat16>(from_f32<__nv_bfloat16>(last));
        float v;
        if (G == 1) {
          v = relu_squared(up);
        } else {
          const float gate = to_f32<__nv_bfloat16>(from_f32<__nv_bfloat16>(sums[t * unit * G + r]));
          if (a.act >= 0) {
            v = glu_activation(gate, a.act) * up;
          } else {
            const float gl = fminf(gate, a.limit);
            v = gl / (1.0f + expf(-a.slope * gl)) * (fminf(fmaxf(up, -a.limit), a.limit) + 1.0f);
          }
        }
        a.y[to] = from_f32<__nv_bfloat16>(v);
      }
      __syncwarp();
      j += unit;
    }
  }
  if (!waited) pdl_wait();  // a block without rows ends no sooner than the kernel before this one
}

// Every token's items, in their order; identity experts hand on the token's row; what a shared expert gave comes last.
__global__ void moe_in_order_sum_kernel(MrArgs p) {
  pdl_launch_dependents();
  pdl_wait();
  const MfArgs& a = p.m;
  const int t = blockIdx.x, c = blockIdx.y * blockDim.x + threadIdx.x;
  if (c >= a.rows) return;
  float total = 0.f;
  for (int k = 0; k < a.top; ++k) {
    const int item = t * a.top + k, e = a.ids[item];
    float d = 0.f;
    if (e >= a.n_real) d = to_f32<__nv_bfloat16>(a.h[(size_t)t * a.rows + c]);
    else if (e >= 0) d = p.d[(size_t)item * a.rows + c];
    const float wt = a.scale_output ? a.weights[item] : 1.0f;
    total += d * wt;
  }
  if (a.add) total += load_as_f32(a.add, a.add_dtype, (size_t)t * a.rows + c) * (a.add_scale ? a.add_scale[t] : 1.0f);
  a.out[(size_t)t * a.rows + c] = total;
}

// Rows of K numbers that fit beside a ring of D stages
static int mr_room(int D, int K, size_t lists) { return (int)((MR_SMEM_MAX - 4096 - mr_ring_bytes(D) - lists) / (2 * (size_t)K)); }

// One product (the launch of an instantiation stands in one place, so that it has one grant): at most `most` tokens of an expert a pass
template <int G, int D>
static int mr_launch(MrArgs& p, int most, size_t lists, cudaStream_t stream) {
  const int room = mr_room(D, p.m.K, lists);
  p.cap = most < room ? most : room;
  if (p.cap < 1) return BN_ERR_BAD_ARG;
  const size_t smem = mr_ring_bytes(D) + (size_t)p.cap * p.m.K * 2 + lists;
  static BnGrant grant;
  cudaError_t e = grant.ask((const void*)moe_in_order_kernel<G, D>, smem, 4096);
  if (e != cudaSuccess) return BN_ERR_LAUNCH + (int)e;
  BN_LAUNCH((moe_in_order_kernel<G, D>), (unsigned)mf_sm_count(), MR_THREADS, smem, stream, p);
  return BN_OK;
}
// Stages: four where the tokens' rows leave room for them, else three.
template <int G>
static int mr_product(MrArgs& p, int most, size_t lists, cudaStream_t stream) {
  return mr_room(4, p.m.K, lists) >= most ? mr_launch<G, 4>(p, most, lists, stream) : mr_launch<G, 3>(p, most, lists, stream);
}

// bn_moe_few with the sums of moe.cu, for the same arguments: d [n_tokens * top, width] float32 is working space.  No row of x may be
// larger than the shared memory beside a ring (width and ff up to 40,960 numbers).
extern "C" int bn_moe_few_in_order(const void* h, int n_tokens, int width, const int* ids, const float* weights, int scale_input, const void* w_gate,
                                   const void* w_up, long long expert_stride, int ff, int top, float limit, float slope, int act, int n_real,
                                   void* y, const void* w_down, const void* add, int add_dtype, const float* add_scale, float* d, float* out,
                                   cudaStream_t stream) {
  if (n_tokens <= 0) return BN_OK;
  if (!h || !ids || !weights || !w_up || !w_down || !y || !d || !out || top <= 0 || top > MF_MAX_ITEMS || n_tokens > MF_MAX_ITEMS / top ||
      n_real <= 0 || n_real > MF_MAX_EXPERTS || width <= 0 || width % 8 || ff <= 0 || ff % 8 || expert_stride % 8 || width > 40960 || ff > 40960 ||
      (((uintptr_t)h | (uintptr_t)w_gate | (uintptr_t)w_up | (uintptr_t)w_down | (uintptr_t)y) & 15))
    return BN_ERR_BAD_ARG;
  MrArgs p = {};
  MfArgs& a = p.m;
  a.x = (const __nv_bfloat16*)h; a.ids = ids; a.weights = weights; a.n_items = n_tokens * top; a.top = top; a.n_real = n_real;
  a.K = width; a.rows = ff; a.w = (const __nv_bfloat16*)w_gate; a.w_up = (const __nv_bfloat16*)w_up; a.expert_stride = (size_t)expert_stride;
  a.scale_input = scale_input; a.limit = limit; a.slope = slope; a.act = act; a.y = (__nv_bfloat16*)y;
  const size_t lists = mf_list_bytes(a) + (3 * a.n_items + 1) * sizeof(int);
  const int most = n_tokens < MR_TOKENS ? n_tokens : MR_TOKENS;
  int rc = w_gate ? mr_product<2>(p, most, lists, stream) : mr_product<1>(p, most, lists, stream);
  if (rc != BN_OK) return rc;
  a.x = (const __nv_bfloat16*)y;
  a.K = ff; a.rows = width; a.w = nullptr; a.w_up = (const __nv_bfloat16*)w_down; a.expert_stride = (size_t)width * ff;
  a.scale_output = !scale_input; a.add = add; a.add_dtype = add_dtype; a.add_scale = add_scale; a.h = (const __nv_bfloat16*)h; a.out = out;
  p.d = d;
  rc = mr_product<1>(p, most, lists, stream);
  if (rc != BN_OK) return rc;
  BN_LAUNCH(moe_in_order_sum_kernel, dim3(n_tokens, (width + 255) / 256), 256, 0, stream, p);
  BN_CHECK_LAUNCH();
  return BN_OK;
}
