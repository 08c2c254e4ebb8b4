// out = act(a . w^T + bias) on the CUDA cores, for any M, N, K.
//
// This is the matrix product of the true 32-bit path (FFMA only: no tensor cores,
// hence no reduced-precision matrix mode) and the fallback of the bfloat16 path
// for shapes the tensor-core kernel refuses.  The weight is [N, K] ("out, in"),
// the layout the reference transposes to at load (crates/core/src/weights.rs:1-9),
// and the product is the reference's x . W^T + b (crates/core/src/kernels/reference.rs:26-37).
//
// The order of an output's sum depends on K alone, never on the other rows of the batch, and is the same in the three
// kernels below: K is cut into segments of 32, each one chain of fused multiply-adds in index order from zero; the
// segments of a quarter of K (whole segments, rounded up) are added in order, and the four quarters are.  Chains of
// 32 instead of one of K make room for many threads an output, and the sum more exact (N(0, 1) values, against 64
// bits, relative: 5.0e-7 -> 1.2e-7 at K = 768, 9.9e-7 -> 1.4e-7 at 3,072).
// Measured on a B200, us, one chain an output with a thread or 4 x 4 outputs of a thread each, and now:
//   rows x N x K:  4 x 768 x 768: 13.7, 3.2     4 x 2304 x 768: 13.7, 4.0    4 x 768 x 3072: 52.6, 7.0
//   4 x 50257 x 768: 57, 34     8 x 50257 x 768: 57, 49     212 x 2304 x 768: 111, 41    212 x 768 x 3072: 229, 54
//   600 x 3072 x 768: 223, 103    2400 x 3072 x 768: 471, 333 (34 TFLOP/s)
#include <atomic>
#include <type_traits>

#include "api.h"
#include "common.cuh"

namespace nib {

constexpr int SEG = 32;        // products in a chain
constexpr int SEG_LD = SEG + 4;   // a segment's pitch in shared memory: eight rows' 16-byte pieces lie in distinct banks

// whole segments in a quarter of K
__host__ __device__ inline int quarter_segments(int K) { return ((K + SEG - 1) / SEG + 3) / 4; }

// Four values of a row from global to shared memory as 32-bit floats: an asynchronous copy where the values are 32-bit
// and the rows 16-byte aligned (VEC), else one by one.  What lies past the row's `K` values, or in a row that is not
// there, is zero.
template <bool VEC, typename T>
__device__ __forceinline__ void stage4(float* dst, const T* row, int k, int K, bool row_ok) {
  if constexpr (VEC) {
    const bool ok = row_ok && k < K;   // (K is a multiple of four)
    cp_async16(dst, ok ? row + k : row, ok);
  } else {
    float v[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) v[i] = row_ok && k + i < K ? to_float(row[k + i]) : 0.0f;
    *reinterpret_cast<float4*>(dst) = make_float4(v[0], v[1], v[2], v[3]);
  }
}

// the chain: acc += a[0] w[0], then a[1] w[1], ...
__device__ __forceinline__ float fma4(float4 a, float4 w, float acc) {
  acc = fmaf(a.x, w.x, acc);
  acc = fmaf(a.y, w.y, acc);
  acc = fmaf(a.z, w.z, acc);
  return fmaf(a.w, w.w, acc);
}

template <typename OutT>
__device__ __forceinline__ void finish(float v, const float* bias, OutT* out, int ldo, int m, int n, int act, int residual) {
  if (bias) v += bias[n];
  v = apply_act(v, act);
  OutT* o = out + (size_t)m * ldo + n;
  if (residual) v += to_float(*o);
  *o = from_float<OutT>(v);
}

// ---------------------------------------------------------------------- more than 16 rows
// A block of 256 threads makes a tile of 16 TM rows x 64 features, TM x 4 outputs a thread, one segment of K at a
// time; the segments come through a ring of shared-memory stages, K running along the rows as in memory, so that
// copies are whole 16-byte pieces and four products of an output need one 16-byte load of each operand.  Bound by the
// multiply-adds and the shared-memory loads that feed them (TM = 4: 8 loads for 64 multiply-adds a thread; eight by
// eight outputs a thread and half the loads were slower up to 600 rows, for want of warps, and 7 % faster beyond).
// Where there are fewer tiles than SMs, a cluster of four blocks takes a quarter of K each and adds the quarters
// through distributed shared memory.
constexpr int TL_N = 64, TL_STAGES = 3;

template <typename InT, typename OutT, int TM, bool VEC>
__global__ void __launch_bounds__(256, 2)
linear_simt_kernel(const InT* a, int lda, const InT* __restrict__ w, int ldw,
                   const float* __restrict__ bias, OutT* out, int ldo, int M, int N,
                   int K, int act, int residual, int split) {
  constexpr int BM = 16 * TM, STAGE = (BM + TL_N) * SEG_LD;
  extern __shared__ __align__(16) float tl_smem[];
  pdl_trigger();
  const int tid = threadIdx.x, tx = tid % 16, ty = tid / 16;   // columns tx + 16 j, rows ty + 16 i
  const int rank = split > 1 ? cluster_rank() : 0;
  const int m0 = blockIdx.y * BM, n0 = (blockIdx.x / split) * TL_N;
  const int n_seg = (K + SEG - 1) / SEG, per_quarter = quarter_segments(K);
  const int seg0 = split > 1 ? rank * per_quarter : 0;
  const int seg1 = split > 1 ? min(n_seg, seg0 + per_quarter) : n_seg;
  const int n_mine = seg1 - seg0;      // (not positive: nothing in this quarter)

  auto ask_w = [&](int i) {            // the weights of this block's segment i: 64 rows of eight pieces
    float* st = tl_smem + (i % TL_STAGES) * STAGE + BM * SEG_LD;
#pragma unroll
    for (int q = 0; q < TL_N * 8 / 256; ++q) {
      const int r = (tid + q * 256) >> 3, c = ((tid + q * 256) & 7) * 4;
      stage4<VEC>(st + r * SEG_LD + c, w + (size_t)min(n0 + r, N - 1) * ldw, (seg0 + i) * SEG + c, K, n0 + r < N);
    }
  };
  auto ask_a = [&](int i) {
    float* st = tl_smem + (i % TL_STAGES) * STAGE;
#pragma unroll
    for (int q = 0; q < (BM * 8 + 255) / 256; ++q) {
      const int r = (tid + q * 256) >> 3, c = ((tid + q * 256) & 7) * 4;
      if (r < BM) stage4<VEC>(st + r * SEG_LD + c, a + (size_t)min(m0 + r, M - 1) * lda, (seg0 + i) * SEG + c, K, m0 + r < M);
    }
  };
  // Without asynchronous copies the next segment waits in registers, a warp loading a row's 32 values at a time, while the
  // one before is used.  us, loads stored at once and now (one chain of K before both): bfloat16, 600 x 9,601 x 1,601 860, 788
  // (755); 200 x 9,601 x 3,073 796, 695 (817); 32 bits, 600 x 9,601 x 1,601 780, 721 (720); 2,000 x 9,601 x 33 107, 89 (69: one value in the
  // second segment); one wave of tiles 0.93 (bfloat16) and 0.99 of the time, at worst 1.07.  Three blocks an SM (80
  // registers) are slower: 844 and 88 for the first and the last.
  const int wr = tid >> 5, wk = tid & 31;
  InT next_w[VEC ? 1 : TL_N / 8], next_a[VEC ? 1 : BM / 8];   // (as they lie in memory: a conversion here would wait)
  auto load_w = [&](int i, InT* v) {
    const int k = (seg0 + i) * SEG + wk;
#pragma unroll
    for (int q = 0; q < TL_N / 8; ++q) {
      const int n = n0 + wr + 8 * q;
      v[q] = n < N && k < K ? w[(size_t)n * ldw + k] : from_float<InT>(0.0f);
    }
  };
  auto load_a = [&](int i, InT* v) {
    const int k = (seg0 + i) * SEG + wk;
#pragma unroll
    for (int q = 0; q < BM / 8; ++q) {
      const int m = m0 + wr + 8 * q;
      v[q] = m < M && k < K ? a[(size_t)m * lda + k] : from_float<InT>(0.0f);
    }
  };
  auto keep = [&](int i, const InT* vw, const InT* va) {
    float* st = tl_smem + (i % TL_STAGES) * STAGE + wr * SEG_LD + wk;
#pragma unroll
    for (int q = 0; q < BM / 8; ++q) st[8 * q * SEG_LD] = to_float(va[q]);
#pragma unroll
    for (int q = 0; q < TL_N / 8; ++q) st[(BM + 8 * q) * SEG_LD] = to_float(vw[q]);
  };
  // the first segments' weights do not depend on the kernel ahead
  if constexpr (VEC) {
#pragma unroll
    for (int i = 0; i < TL_STAGES - 1; ++i)
      if (i < n_mine) ask_w(i);
    pdl_wait();
#pragma unroll
    for (int i = 0; i < TL_STAGES - 1; ++i) {
      if (i < n_mine) ask_a(i);
      cp_async_commit();
    }
  } else {
    InT first_w[TL_N / 8], first_a[BM / 8];
    if (n_mine > 0) load_w(0, first_w);
    if (n_mine > 1) load_w(1, next_w);
    pdl_wait();
    if (n_mine > 0) load_a(0, first_a);
    if (n_mine > 1) load_a(1, next_a);
    if (n_mine > 0) keep(0, first_w, first_a);
  }
  float total[TM][4], quarter[TM][4];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) total[i][j] = quarter[i][j] = 0.0f;

  for (int s = 0; s < n_mine; ++s) {
    if constexpr (VEC) cp_async_wait<TL_STAGES - 2>();    // (one group a segment, empty ones at the end)
    __syncthreads();                   // segment s is there for all, and segment s - 1 has been used by all
    if constexpr (VEC) {
      if (s + TL_STAGES - 1 < n_mine) {
        ask_w(s + TL_STAGES - 1);
        ask_a(s + TL_STAGES - 1);
      }
      cp_async_commit();
    } else {
      if (s + 1 < n_mine) keep(s + 1, next_w, next_a);
      if (s + 2 < n_mine) {
        load_w(s + 2, next_w);
        load_a(s + 2, next_a);
      }
    }
    const float* as = tl_smem + (s % TL_STAGES) * STAGE + ty * SEG_LD;
    const float* ws = tl_smem + (s % TL_STAGES) * STAGE + (BM + tx) * SEG_LD;
    float acc[TM][4];
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) acc[i][j] = 0.0f;
    auto step = [&](int k) {
      float4 av[TM], wv[4];
#pragma unroll
      for (int i = 0; i < TM; ++i) av[i] = *reinterpret_cast<const float4*>(as + i * 16 * SEG_LD + k);
#pragma unroll
      for (int j = 0; j < 4; ++j) wv[j] = *reinterpret_cast<const float4*>(ws + j * 16 * SEG_LD + k);
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = fma4(av[i], wv[j], acc[i][j]);
    };
    const int left = VEC ? SEG : K - (seg0 + s) * SEG;    // (the zeros past the end of an odd K are left out)
    if (left >= SEG) {
#pragma unroll
      for (int k = 0; k < SEG; k += 4) step(k);
    } else {
#pragma unroll 1
      for (int k = 0; k < left; k += 4) step(k);
    }
    const bool quarter_ends = (seg0 + s + 1) % per_quarter == 0 || s + 1 == n_mine;
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        quarter[i][j] += acc[i][j];
        if (quarter_ends) {
          total[i][j] += quarter[i][j];
          quarter[i][j] = 0.0f;
        }
      }
  }
  if (split > 1) {
    // every block leaves its quarter's sums in its own shared memory; block r of the cluster then adds up and
    // finishes the outputs with i % 4 == r, in the order of the quarters
    cp_async_wait<0>();
    __syncthreads();
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) tl_smem[(i * 4 + j) * 256 + tid] = total[i][j];
    cluster_arrive();
    cluster_wait();
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int m = m0 + ty + 16 * i, n = n0 + tx + 16 * j;
        if (j != rank || m >= M || n >= N) continue;
        float v = 0.0f;
        for (int q = 0; q < 4; ++q) v += __uint_as_float(cluster_load(cluster_addr(tl_smem + (i * 4 + j) * 256 + tid, q)));
        finish(v, bias, out, ldo, m, n, act, residual);
      }
    cluster_arrive();                  // nobody leaves while another block still reads here
    cluster_wait();
    return;
  }
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int m = m0 + ty + 16 * i, n = n0 + tx + 16 * j;
      if (m < M && n < N) finish(total[i][j], bias, out, ldo, m, n, act, residual);
    }
}

// ---------------------------------------------------------------------- at most 16 rows
// A decode step is a stream of weights.  A block makes eight features at a time; of up to 1,024 of K at a time, every
// thread takes one feature's segment of 32 for all rows, so that a product of 768 x 768 occupies 24,576 threads.
// Weights and rows come by asynchronous copies of whole 16-byte pieces, the next ones while these are used; the
// segments' sums meet in shared memory, where one thread an output adds them in order.  A wide output (the head) is
// walked by as many blocks as the device holds, which read the step's rows once where K fits a stage (reading them
// for every eight features doubles what an SM takes in at eight rows).  Bound by the memory there, and for the narrow
// products by the chain copy -> chains of 32 -> sums.
constexpr int RW_F = 8, RW_SEGS = 32, RW_K = RW_SEGS * SEG;

// a row's pitch in a stage; a feature's is 4 more, so that eight features lie in distinct banks (K of 768: 24 segments)
__host__ __device__ inline int rows_pitch(int K) {
  const int n = (K + SEG - 1) / SEG;
  const int segs = n < RW_SEGS ? (n + 7) / 8 * 8 : RW_SEGS;   // (a multiple of 32 floats)
  return segs * SEG_LD;
}

// the segments' sums: behind the stages, or, for 16 rows, which leave no room, over the weights that were just used
template <int ROWS>
static constexpr bool rows_alias = ROWS > 8;
// w_stages, a_stages: 1 or 2 stages of weights, and of rows
template <int ROWS>
static size_t rows_smem(int w_stages, int a_stages, int K) {
  const size_t ld = rows_pitch(K);
  return sizeof(float) * (w_stages * RW_F * (ld + 4) + a_stages * ROWS * ld + (rows_alias<ROWS> ? 0 : ld / SEG_LD * RW_F * ROWS));
}

// (`a` and `out` carry no __restrict__: see pdl_wait in common.cuh.  With it, the compiler read the
// step's rows beside the weights, above the wait, before the kernel that writes them had finished.)
template <typename InT, typename OutT, int ROWS, bool VEC>
__global__ void __launch_bounds__(256)
linear_simt_rows_kernel(const InT* a, int lda, const InT* __restrict__ w, int ldw,
                        const float* __restrict__ bias, OutT* out, int ldo, int M, int N, int K,
                        int act, int residual, int w_stages) {
  constexpr bool ALIAS = rows_alias<ROWS>;
  const int A_LD = rows_pitch(K), W_LD = A_LD + 4, RW_W = RW_F * W_LD;
  extern __shared__ __align__(16) float rw_smem[];
  pdl_trigger();
  const int tid = threadIdx.x;
  const int f = tid & (RW_F - 1), sg = tid / RW_F;   // this thread's feature and segment
  const int n_seg = (K + SEG - 1) / SEG, per_quarter = quarter_segments(K);
  const int n_st = (n_seg + RW_SEGS - 1) / RW_SEGS;  // stages of K
  const int a_stages = min(n_st, 2);
  const int n_groups = (N + RW_F - 1) / RW_F;        // of eight features; this block's are blockIdx.x + i * gridDim.x
  const int n_it = ((n_groups - 1 - (int)blockIdx.x) / (int)gridDim.x + 1) * n_st;
  float* a_smem = rw_smem + w_stages * RW_W;
  // round `it` is stage `st` of group `g` (of this block's); its weights go to buffer it % w_stages, its rows to it % a_stages
  auto ask_w = [&](int it, int st, int g) {          // 256 pieces of each feature's row; those past K's end are not made
    const int k = st * RW_K + tid * 4, n0 = ((int)blockIdx.x + g * (int)gridDim.x) * RW_F;
    if (k >= n_seg * SEG) return;
    float* dst = rw_smem + (it & (w_stages - 1)) * RW_W + (tid >> 3) * SEG_LD + (tid & 7) * 4;
#pragma unroll
    for (int r = 0; r < RW_F; ++r) stage4<VEC>(dst + r * W_LD, w + (size_t)min(n0 + r, N - 1) * ldw, k, K, n0 + r < N);
  };
  auto ask_a = [&](int it, int st) {                 // (where K fits a stage, the rows stay)
    const int k = st * RW_K + tid * 4;
    if (k >= n_seg * SEG || (n_st == 1 && it > 0)) return;
    float* dst = a_smem + (it & (a_stages - 1)) * ROWS * A_LD + (tid >> 3) * SEG_LD + (tid & 7) * 4;
#pragma unroll
    for (int r = 0; r < ROWS; ++r) stage4<VEC>(dst + r * A_LD, a + (size_t)min(r, M - 1) * lda, k, K, r < M);
  };
  int st_ahead = 0, g_ahead = 0;                     // stage and group of the next round to ask for
  auto advance = [&]() { if (++st_ahead == n_st) { st_ahead = 0; ++g_ahead; } };
  constexpr int PARTS = (RW_F * ROWS * 4 + 255) / 256;
  // What a sum meets at its end is asked for with the group's first stage: the bias ahead of the wait, the old value of a
  // residual output with the rows.  (Asked for at the end, one behind the other, they were two round trips to L2; with the
  // divisions of a round's number gone as well, a launch of 4 rows in a step of GPT-2 small 5.65 -> 4.9 us.)
  float quarter[PARTS], bias_r[PARTS], res_r[PARTS];
  auto mine = [&](int p, int g, int& m, int& n) {    // output p of this thread in group g
    const int o = (tid >> 2) + p * 64;
    m = o % ROWS;
    n = ((int)blockIdx.x + g * (int)gridDim.x) * RW_F + o / ROWS;
    return (tid & 3) == 0 && (RW_F * ROWS >= 64 || o < RW_F * ROWS) && m < M && n < N;
  };
  auto ask_bias = [&](int g) {
#pragma unroll
    for (int p = 0; p < PARTS; ++p) {
      int m, n;
      bias_r[p] = bias != nullptr && mine(p, g, m, n) ? bias[n] : 0.0f;
    }
  };
  auto ask_residual = [&](int g) {
#pragma unroll
    for (int p = 0; p < PARTS; ++p) {
      int m, n;
      res_r[p] = residual && mine(p, g, m, n) ? to_float(out[(size_t)m * ldo + n]) : 0.0f;
    }
  };
  ask_w(0, 0, 0);
  advance();
  if (n_it > 1 && w_stages > 1) ask_w(1, st_ahead, g_ahead);
  ask_bias(0);
  pdl_wait();
  ask_a(0, 0);
  cp_async_commit();
  if (n_it > 1 && w_stages > 1) ask_a(1, st_ahead);
  cp_async_commit();
  advance();
  ask_residual(0);
  int st = 0, g = 0;
#pragma unroll
  for (int p = 0; p < PARTS; ++p) quarter[p] = 0.0f;
  for (int it = 0; it < n_it; ++it) {
    cp_async_wait<1>();                              // (one group a round, empty ones at the end)
    __syncthreads();
    const int segs = min(RW_SEGS, n_seg - st * RW_SEGS);
    float acc[ROWS];
    if (sg < segs) {
      const float* ws = rw_smem + (it & (w_stages - 1)) * RW_W + f * W_LD + sg * SEG_LD;
      const float* as = a_smem + (it & (a_stages - 1)) * ROWS * A_LD + sg * SEG_LD;
#pragma unroll
      for (int r = 0; r < ROWS; ++r) acc[r] = 0.0f;
#pragma unroll
      for (int k = 0; k < SEG; k += 4) {
        const float4 wv = *reinterpret_cast<const float4*>(ws + k);
#pragma unroll
        for (int r = 0; r < ROWS; ++r) acc[r] = fma4(*reinterpret_cast<const float4*>(as + r * A_LD + k), wv, acc[r]);
      }
    }
    // [segment][feature][row]
    float* red = ALIAS ? rw_smem + (it & (w_stages - 1)) * RW_W : a_smem + a_stages * ROWS * A_LD;
    if (ALIAS) __syncthreads();
    if (sg < segs) {
#pragma unroll
      for (int r = 0; r < ROWS; ++r) red[(sg * RW_F + f) * ROWS + r] = acc[r];
    }
    __syncthreads();                                 // the stage has been used, its sums are there
    if (!ALIAS && it + 2 < n_it) {
      ask_w(it + 2, st_ahead, g_ahead);
      ask_a(it + 2, st_ahead);
    }
    if (!ALIAS) cp_async_commit();
    // the quarters of an output side by side in four lanes: each adds its segments of this stage, in order
#pragma unroll
    for (int p = 0; p < PARTS; ++p) {
      const int o = (tid >> 2) + p * 64, q = tid & 3;      // output (feature o / ROWS, row o % ROWS), quarter
      if (RW_F * ROWS >= 64 || o < RW_F * ROWS) {          // (whole warps)
        const int i1 = min(segs, (q + 1) * per_quarter - st * RW_SEGS);
#pragma unroll 4
        for (int i = max(0, q * per_quarter - st * RW_SEGS); i < i1; ++i) quarter[p] += red[i * RW_F * ROWS + o];
        if (st + 1 == n_st) {
          float total = quarter[p];
          total += __shfl_down_sync(0xffffffffu, quarter[p], 1, 4);
          total += __shfl_down_sync(0xffffffffu, quarter[p], 2, 4);
          total += __shfl_down_sync(0xffffffffu, quarter[p], 3, 4);
          int m, n;
          if (mine(p, g, m, n)) {
            float v = apply_act(total + bias_r[p], act);
            if (residual) v += res_r[p];
            out[(size_t)m * ldo + n] = from_float<OutT>(v);
          }
          quarter[p] = 0.0f;
        }
      }
    }
    if (ALIAS) {
      __syncthreads();
      if (it + 2 < n_it) {
        ask_w(it + 2, st_ahead, g_ahead);
        ask_a(it + 2, st_ahead);
      }
      cp_async_commit();
    }
    advance();
    if (++st == n_st) {
      st = 0;
      ++g;
      if (it + 1 < n_it) {
        ask_bias(g);
        ask_residual(g);
      }
    }
  }
}

// ---------------------------------------------------------------------- at most 16 rows and few chunks of K
// With K of one or two hundred a block of the kernel above has segments for a few of its threads only, and a wide output
// many blocks.  Here a block owns 64 features and every thread one feature for ROWS / 4 of the step's rows; K comes in
// chunks of 64 that are asked for two chunks ahead (registers).  A chunk costs about 1.05 us whatever the rows (1.35 with
// 16 rows) while a block has an SM to itself: a chain of round trips, and bound by it.
constexpr int FB_N = 64, FB_K = 2 * SEG;

template <typename InT, typename OutT, int ROWS>
__global__ void __launch_bounds__(256)
linear_simt_features_kernel(const InT* a, int lda, const InT* __restrict__ w, int ldw,
                            const float* __restrict__ bias, OutT* out, int ldo, int M, int N, int K,
                            int act, int residual) {
  constexpr int RPT = ROWS / 4;                      // rows per thread
  constexpr int WPT = FB_N * FB_K / 256;             // weight values a thread stages per chunk: 16
  constexpr int APT = (ROWS * FB_K + 255) / 256;     // values of the step's rows per thread and chunk
  pdl_trigger();
  __shared__ float Ws[2][FB_N][FB_K + 1];
  __shared__ __align__(16) float As[2][ROWS][FB_K];
  const int tid = threadIdx.x, n0 = blockIdx.x * FB_N;
  const int f = tid % FB_N, rg = tid / FB_N;
  const int lk = tid % FB_K, lr = tid / FB_K;        // staging: column of the chunk, first of the rows (step 4)
  const int per_quarter = quarter_segments(K);
  int left = per_quarter;                            // segments until the quarter ends
  float wreg[2][WPT], areg[2][APT];
  // asks for chunk c (columns c * 64 ...) into the register set `s`: weights do not depend on the kernel
  // ahead, the step's rows do
  auto ask_w = [&](int c, int s) {
#pragma unroll
    for (int j = 0; j < WPT; ++j) {
      const int n = n0 + lr + 4 * j, k = c * FB_K + lk;
      wreg[s][j] = (n < N && k < K) ? to_float(w[(size_t)n * ldw + k]) : 0.0f;
    }
  };
  auto ask_a = [&](int c, int s) {
#pragma unroll
    for (int j = 0; j < APT; ++j) {
      const int m = lr + 4 * j, k = c * FB_K + lk;
      areg[s][j] = (m < M && m < ROWS && k < K) ? to_float(a[(size_t)m * lda + k]) : 0.0f;
    }
  };
  const int n_chunks = (K + FB_K - 1) / FB_K;
  ask_w(0, 0);
  if (n_chunks > 1) ask_w(1, 1);
  pdl_wait();
  ask_a(0, 0);
  if (n_chunks > 1) ask_a(1, 1);
  float total[RPT], quarter[RPT];
#pragma unroll
  for (int i = 0; i < RPT; ++i) total[i] = quarter[i] = 0.0f;
  // one chunk: the registers of set S go to buffer S, the chunk after next is asked for into them, and
  // the chunk's two segments are added (S is a constant of the code, so that the sets stay in registers)
  auto chunk = [&](int c, auto S) {
    constexpr int s = decltype(S)::value;
#pragma unroll
    for (int j = 0; j < WPT; ++j) Ws[s][lr + 4 * j][lk] = wreg[s][j];
#pragma unroll
    for (int j = 0; j < APT; ++j) As[s][lr + 4 * j][lk] = areg[s][j];
    if (c + 2 < n_chunks) {
      ask_w(c + 2, s);
      ask_a(c + 2, s);
    }
    __syncthreads();          // (two buffers by turns: a buffer is written again two chunks later, a barrier between)
    float acc[2][RPT];        // the chunk's two segments (past the end of K: zeros, which change nothing)
#pragma unroll
    for (int i = 0; i < RPT; ++i) acc[0][i] = acc[1][i] = 0.0f;
#pragma unroll 2
    for (int k = 0; k < SEG; k += 4) {
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const float* ws = &Ws[s][f][h * SEG + k];
        const float4 wv = make_float4(ws[0], ws[1], ws[2], ws[3]);
#pragma unroll
        for (int i = 0; i < RPT; ++i)
          acc[h][i] = fma4(*reinterpret_cast<const float4*>(&As[s][rg * RPT + i][h * SEG + k]), wv, acc[h][i]);
      }
    }
#pragma unroll
    for (int h = 0; h < 2; ++h) {
#pragma unroll
      for (int i = 0; i < RPT; ++i) quarter[i] += acc[h][i];
      if (--left == 0) {
#pragma unroll
        for (int i = 0; i < RPT; ++i) {
          total[i] += quarter[i];
          quarter[i] = 0.0f;
        }
        left = per_quarter;
      }
    }
  };
  for (int c = 0; c < n_chunks; c += 2) {
    chunk(c, std::integral_constant<int, 0>());
    if (c + 1 < n_chunks) chunk(c + 1, std::integral_constant<int, 1>());
  }
  const int n = n0 + f;
  if (n >= N) return;
#pragma unroll
  for (int i = 0; i < RPT; ++i) {
    const int m = rg * RPT + i;
    if (m < M) finish(total[i] + quarter[i], bias, out, ldo, m, n, act, residual);
  }
}

template <typename K>
static cudaError_t allow_smem(K kernel, size_t bytes) {
  return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
}

template <typename InT, typename OutT, int ROWS, bool VEC>
static int launch_rows(const InT* a, int lda, const InT* w, int ldw, const float* bias, OutT* out, int ldo, int M, int N,
                       int K, int act, int residual, cudaStream_t stream) {
  auto kernel = linear_simt_rows_kernel<InT, OutT, ROWS, VEC>;
  static const cudaError_t allowed = allow_smem(kernel, rows_smem<ROWS>(2, 2, 2 * RW_K));
  if (allowed != cudaSuccess) return (int)allowed;
  const int n_st = (K + RW_K - 1) / RW_K, a_stages = n_st < 2 ? 1 : 2, groups = (N + RW_F - 1) / RW_F;
  // One group of features a block while the device holds them all at once (a block that has one round needs one stage
  // of weights); else as many blocks as it holds, with two stages.  What an SM holds is asked for once for each size of a
  // stage (registers count too: with 8 and 16 rows they leave room for two blocks).
  cudaError_t err = cudaSuccess;
  auto held = [&](int w_stages) {
    static std::atomic<int> kept[5][2];      // [eighths of a stage that K fills, less one; several stages][stages of weights]
    std::atomic<int>& slot = kept[n_st > 1 ? 4 : rows_pitch(K) / (8 * SEG_LD) - 1][w_stages - 1];
    int n = slot.load(std::memory_order_relaxed);
    if (n == 0) {
      err = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kernel, 256, rows_smem<ROWS>(w_stages, a_stages, K));
      if (err != cudaSuccess) return 148;
      slot.store(n = n < 1 ? 1 : n, std::memory_order_relaxed);
    }
    return 148 * n;
  };
  int w_stages = n_st > 1 ? 2 : 1, blocks = groups;
  if (groups > held(w_stages)) {
    w_stages = 2;
    blocks = held(2);
  }
  if (err != cudaSuccess) return (int)err;
  launch_pdl(kernel, dim3(blocks), dim3(256), rows_smem<ROWS>(w_stages, a_stages, K), stream, a, lda, w, ldw, bias, out, ldo, M,
             N, K, act, residual, w_stages);
  NIB_LAUNCH_CHECK();
}

template <typename InT, typename OutT, int ROWS, bool VEC>
static int launch_features(const InT* a, int lda, const InT* w, int ldw, const float* bias, OutT* out, int ldo, int M, int N,
                           int K, int act, int residual, cudaStream_t stream) {
  launch_pdl(linear_simt_features_kernel<InT, OutT, ROWS>, dim3((N + FB_N - 1) / FB_N), dim3(256), 0, stream, a, lda, w, ldw,
             bias, out, ldo, M, N, K, act, residual);
  NIB_LAUNCH_CHECK();
}

// Up to how many chunks of K (64) the kernel above is ahead.  It costs about a chunk's round trip a chunk; the other one
// about the same whatever K up to several hundred, but a group of eight features at a time, so that it falls behind where
// outputs are wide or rows many; without asynchronous copies (16-bit values, odd pitches) sooner.  us, this one and the
// other: N = 768, K = 64: 1 row 1.80, 1.91, 16 rows 2.45, 3.00; K = 128, 16 rows 3.46, 3.11.  N = 3,072: K = 128, 4 rows 2.86,
// 3.35, 16 rows 3.52, 5.58; K = 256, 16 rows 6.31, 6.05.  N = 9,600: K = 64, 8 rows 3.05, 6.76; K = 128, 1 row 4.29, 3.86, 4 rows
// 4.39, 5.01; K = 256, 8 rows 9.32, 7.57, 16 rows 9.87, 12.34; K = 384, 16 rows 14.4, 13.6.  N = 50,257, K = 768, 16 rows 83, 86.
// bfloat16: N = 768, K = 33: 8 rows 2.12, 3.67; K = 100: 4 rows 2.96, 2.41, 8 rows 3.00, 3.60; N = 9,600, K = 130: 8 rows 7.24, 10.07.
// From how many features on it is ahead whatever K: the other kernel's time grows with their number, and where K takes
// several stages it reads the rows again for every eight of them; without asynchronous copies it waits for every stage.
// us, this one and the other, 16 rows, 32-bit: K = 768: N = 9,601 28, 20; 14,400 28, 27; 18,944 28, 35.  K = 1,600: 8,192 53, 48;
// 12,288 58, 73; 18,944 59, 108; 50,257 173, 284.  8 rows: K = 768, 50,257 59, 49; K = 1,600: 14,400 62, 49; 18,944 45, 62; 50,257
// 123, 161.  Odd pitches, 16 rows: K = 769: 8,192 28, 26; 9,601 30, 32; K = 1,601: 5,120 52, 47; 6,144 42, 56; 8 rows: K = 769:
// 14,400 32, 28; 18,944 23, 36; K = 1,601: 9,601 59, 50; 12,288 57, 66; 4 rows, K = 1,601: 14,400 64, 47; 18,944 46, 60.  bfloat16, 16
// rows: K = 769: 9,601 42, 37; 12,288 42, 46; K = 1,601: 6,144 79, 78; 7,168 82, 90; 8 rows: K = 769: 12,288 36, 33; 14,400 36, 39;
// K = 1,601: 9,601 69, 67; 12,288 71, 87; 4 rows: behind up to 50,257.
template <typename InT, bool VEC>
static bool features_pay(int M, int N, int K) {
  const bool wide = N >= 8192, middle = N >= 2048, half = sizeof(InT) == 2, stages = K > RW_K;
  int most;
  if (M <= 2) most = half && wide ? 2 : 1;
  else if (M <= 4) most = wide || (middle && (VEC || half)) ? 2 : 1;
  else if (M <= 8) most = half ? (wide ? 3 : 2) : VEC ? (N >= 16384 ? 4 : wide ? 3 : middle ? 2 : 1) : wide ? 2 : 1;
  else most = wide ? 5 : middle ? 3 : VEC ? 1 : 2;
  if ((K + FB_K - 1) / FB_K <= most) return true;
  if (M <= 4) return !VEC && !half && stages && N >= 16384;
  if (M <= 8) return VEC ? stages && N >= 16384 : N >= (stages ? 12288 : half ? 14336 : 16384);
  return N >= (VEC ? (stages ? 12288 : 16384) : half ? (stages ? 7168 : 12288) : (stages ? 6144 : 9216));
}

template <typename InT, typename OutT, int TM, bool VEC>
static int launch_tile(const InT* a, int lda, const InT* w, int ldw, const float* bias, OutT* out, int ldo, int M, int N,
                       int K, int act, int residual, cudaStream_t stream) {
  constexpr size_t smem = sizeof(float) * TL_STAGES * (16 * TM + TL_N) * SEG_LD;
  auto kernel = linear_simt_kernel<InT, OutT, TM, VEC>;
  static const cudaError_t allowed = allow_smem(kernel, smem);
  if (allowed != cudaSuccess) return (int)allowed;
  const int nx = (N + TL_N - 1) / TL_N, ny = (M + 16 * TM - 1) / (16 * TM);
  // fewer tiles than SMs: four blocks a tile, a quarter of K each (from two segments a quarter on)
  const int split = (long)nx * ny <= 148 && quarter_segments(K) >= 2 ? 4 : 1;
  launch_pdl_cluster(kernel, dim3(nx * split, ny), dim3(256), smem, stream, split, a, lda, w, ldw, bias, out, ldo, M, N, K, act,
                     residual, split);
  NIB_LAUNCH_CHECK();
}

template <typename InT, typename OutT, bool VEC>
static int launch_any(const InT* a, int lda, const InT* w, int ldw, const float* bias, OutT* out, int ldo, int M, int N,
                      int K, int act, int residual, cudaStream_t stream) {
#define NIB_SIMT(F, P) F<InT, OutT, P, VEC>(a, lda, w, ldw, bias, out, ldo, M, N, K, act, residual, stream)
  if (M <= 16 && features_pay<InT, VEC>(M, N, K)) return M <= 8 ? NIB_SIMT(launch_features, 8) : NIB_SIMT(launch_features, 16);
  if (M <= 2) return NIB_SIMT(launch_rows, 2);
  if (M <= 4) return NIB_SIMT(launch_rows, 4);
  if (M <= 8) return NIB_SIMT(launch_rows, 8);
  if (M <= 16) return NIB_SIMT(launch_rows, 16);
  // tiles of 32 rows where they waste less: up to 32 rows, and 65 to 96
  if (M <= 32 || (M > 64 && M <= 96)) return NIB_SIMT(launch_tile, 2);
  return NIB_SIMT(launch_tile, 4);
#undef NIB_SIMT
}

template <typename InT, typename OutT>
static int launch(const void* a, int lda, const void* w, int ldw, const float* bias, void* out, int ldo, int M, int N, int K,
                  int act, int residual, cudaStream_t stream) {
  // asynchronous copies want 32-bit values in 16-byte pieces: K, row pitches and addresses all multiples of four values
  if constexpr (sizeof(InT) == 4) {
    if (K % 4 == 0 && lda % 4 == 0 && ldw % 4 == 0 && (((uintptr_t)a | (uintptr_t)w) & 15) == 0)
      return launch_any<InT, OutT, true>((const InT*)a, lda, (const InT*)w, ldw, bias, (OutT*)out, ldo, M, N, K, act, residual,
                                         stream);
  }
  return launch_any<InT, OutT, false>((const InT*)a, lda, (const InT*)w, ldw, bias, (OutT*)out, ldo, M, N, K, act, residual,
                                      stream);
}

}  // namespace nib

using namespace nib;

extern "C" int nib_linear_simt(int in_dtype, int out_dtype, const void* a, int lda, const void* w,
                               int ldw, const float* bias, void* out, int ldo, int M, int N, int K,
                               int act, int residual, cudaStream_t stream) {
  if (M <= 0 || N <= 0) return 0;
  if (K <= 0) return NIB_ERR_BAD_ARGUMENT;
  if (residual && out_dtype != DT_F32) return NIB_ERR_BAD_ARGUMENT;  // the residual stream is 32-bit
  if ((M + 63) / 64 > 65535) return NIB_ERR_UNSUPPORTED_SIZE;
  if (in_dtype == DT_F32 && out_dtype == DT_F32)
    return launch<float, float>(a, lda, w, ldw, bias, out, ldo, M, N, K, act, residual, stream);
  if (in_dtype == DT_BF16 && out_dtype == DT_BF16)
    return launch<bf16, bf16>(a, lda, w, ldw, bias, out, ldo, M, N, K, act, residual, stream);
  if (in_dtype == DT_BF16 && out_dtype == DT_F32)
    return launch<bf16, float>(a, lda, w, ldw, bias, out, ldo, M, N, K, act, residual, stream);
  return NIB_ERR_BAD_ARGUMENT;
}
