// Plain matrix product on the ordinary arithmetic units (no reduced precision): the
// yardstick the bfloat16 tensor-core kernels are tested against, and the matrix product of
// the 32-bit path where w's rows are short, its outputs very wide, or rows come in batches
// and groups.  (Other 32-bit products run on the tensor cores, operands cut in three, gemm_f32.cuh.)
//
//   out[m, n] = OutT( sum_k x[m, k] * w[n, k]  (+ bias[n]) )          w is [out, in]
//   gated:      out[m, n] = T( silu(g) * u ),  g = x . w[n], u = x . w[inter + n]   (32-bit, one rounding)
//
// The sum over k is taken in four parts: blocks of 16 k's go to the parts in turn, a part
// runs over its blocks in ascending order, even and odd k's apart, with one fused
// multiply-add per term; a part is even + odd, the parts are added as (0 + 1) + (2 + 3).
// The kernel for few rows and the tiles take it so, whatever the number of rows: an output
// element does not depend on how the rows were batched.  (Two kernels for few rows take lanes
// over k and a shuffle tree: a batch of heads of up to 16 rows, and grouped rows of a decode
// step.  Their elements differ from the tiles' by 32-bit roundings.)  Formulas:
// rust/engine/src/runner/model/qwen2/kernels.rs:156-178, 393-418 (linear, bias in 32-bit,
// one rounding), 422-448 (gate/up with the SiLU product), 1469-1486 (SiLU).
#include <type_traits>

#include "gemm_f32.cuh"

namespace {
constexpr int BM = 64;      // rows of a group's tiles in the layout of grouped rows
constexpr int PARTS = 4, PART_K = 16, STAGE_K = PARTS * PART_K;      // how the sum over k is cut (see the top)

// 16 (or 4) bytes, zeros where `has` is false, from global to shared memory without a register in between.
__device__ __forceinline__ void cp_async16(void* dst, const void* src, bool has) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(dst)), "l"(src), "r"(has ? 16 : 0)
               : "memory");
}
__device__ __forceinline__ void cp_async4(void* dst, const void* src, bool has) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(smem_u32(dst)), "l"(src), "r"(has ? 4 : 0) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// Two products at once, the sums of even and of odd k's: an instruction reads its operands as the pairs in which they
// lie in memory.
struct Quad {
  unsigned long long lo, hi;
};
__device__ __forceinline__ float sum_of_pair(f32x2 d) { return low_of(d) + high_of(d); }
__device__ __forceinline__ Quad load_quad(const float* p) {
  const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(p);
  return {v.x, v.y};
}
__device__ __forceinline__ Quad load_quad(const __nv_bfloat16* p) {
  const float4 v = load4(p);
  Quad q;
  asm("mov.b64 %0, {%1, %2};" : "=l"(q.lo) : "f"(v.x), "f"(v.y));
  asm("mov.b64 %0, {%1, %2};" : "=l"(q.hi) : "f"(v.z), "f"(v.w));
  return q;
}

// A tile of 4 MI rows by 64 columns (gated: 32 gate columns and the same up columns of w), a warp for each part of the
// sum over k, all on the same tile; their sums are added at the end.  A warp's lanes lie 4 x 8 over the tile; a lane
// keeps MI rows, 4 apart, by 8 columns, 8 apart.
//
// What bounds it: multiply-adds, of which a warp's 8 x 8 products a lane reach half of the units' rate (37 of 74
// TFLOP/s, the pipe 51 % busy, six warps a multiprocessor that wait for their own results; larger tiles a lane or a CTA,
// one multiply-add an instruction, or more warps a multiprocessor did not pass that).  The four warps are what spreads an
// output of few tiles over the multiprocessors' four schedulers.  Operands lie in shared memory as they lie in memory,
// row by row, rows an odd number of 16-byte units apart (no bank conflicts), and come by cp.async through a ring of
// STAGES stages of 64 k's: copies in flight cost no registers and are waited for in their order.  VEC: rows are whole
// 16-byte units; else elements are copied one by one.
// Measured on a B200, 32-bit, weights from memory, against tiles of 64 x 64 by one sum over k, loaded 16 k's at a time:
// 517 x 4864 x 896 gated 263 us (349), 517 x 896 x 4864 155 us (509), 100 x 896 x 4864 64 us (413).
template <typename T, int MI> struct TileShape {
  static constexpr int ROWS = 4 * MI, COLS = 64, THREADS = PARTS * 32;
  static constexpr int UNIT = 16 / (int)sizeof(T), LD = STAGE_K + UNIT;      // elements of 16 bytes, and between rows
  static constexpr int STAGES = 3;
  static constexpr int RING = (int)sizeof(T) * STAGES * LD * (ROWS + COLS);
  static constexpr int SUMS = 2 * 4 * MI * 8 * 32;         // two warps' sums, for the end
  static constexpr int BYTES = RING > SUMS ? RING : SUMS;
};

template <typename T, typename OutT, bool GATED, int MI, bool VEC>
__global__ void __launch_bounds__(PARTS * 32) gemm_plain_kernel(
    OutT* __restrict__ out, const T* __restrict__ x, const T* __restrict__ w, const T* __restrict__ bias, int M, int N,
    int K, int ldx, int ldo, long long batch_x, long long batch_w, long long batch_o, int gelu,
    const int* __restrict__ row_src, int row_div, const int* __restrict__ tile_group, int gate_act, float gate_limit,
    const float* __restrict__ row_scale) {
  using Shape = TileShape<T, MI>;
  constexpr int TM = Shape::ROWS, TN = Shape::COLS, NT = Shape::THREADS, LD = Shape::LD, UNIT = Shape::UNIT;
  constexpr int STAGES = Shape::STAGES, ROWS = TM + TN, UNITS = STAGE_K / UNIT;      // rows of a stage: x's, then w's
  constexpr int STEP = NT / UNITS, COPIES = ROWS / STEP;      // a thread's copies lie STEP rows apart
  constexpr int OUT_N = GATED ? TN / 2 : TN;
  static_assert(ROWS % STEP == 0, "every thread copies alike");
  extern __shared__ __align__(16) char gp_smem[];
  T* smem = reinterpret_cast<T*>(gp_smem);
  pdl_wait();
  // a batch of products of one shape (blockIdx.z): operand b lies b * batch_* elements further on
  x += blockIdx.z * batch_x;
  w += blockIdx.z * batch_w;
  out += blockIdx.z * batch_o;
  // grouped rows: every BM rows meet the matrix of their own group (tile_group[row / BM], -1: a tile without
  // rows), batch_w elements apart; row m reads x's row row_src[m] / row_div (-1: a row of padding, zeros)
  if (tile_group != nullptr) {
    const int group = tile_group[blockIdx.y * TM / BM];
    if (group < 0) return;
    w += (long long)group * batch_w;
  }
  const int tid = threadIdx.x, lane = tid & 31, part = tid >> 5;
  const int m0 = blockIdx.y * TM, n0 = blockIdx.x * OUT_N;

  // where each row of a stage lies in memory; rows and columns beyond the last (null) are zeros
  __shared__ const T* src[ROWS];
  for (int row = tid; row < ROWS; row += NT) {
    const T* at = nullptr;
    if (row < TM) {
      int m = m0 + row;
      if (m < M && row_src != nullptr) {
        m = row_src[m];
        m = m < 0 ? M : m / row_div;
        if (m != M) at = x + (size_t)m * ldx;
      } else if (m < M) {
        at = x + (size_t)m * ldx;
      }
    } else {
      const int c = row - TM, n = n0 + (GATED ? c % 32 : c);      // gated: 32 gate columns, then their up columns
      if (n < N) at = w + (size_t)(GATED && c >= 32 ? N + n : n) * K;
    }
    src[row] = at;
  }
  __syncthreads();
  const int unit = tid % UNITS, first = tid / UNITS;      // a thread copies one unit of every STEP-th row
  const int stages = (K + STAGE_K - 1) / STAGE_K;
  auto fetch = [&](int s) {
    if (s < stages) {
      const int k = s * STAGE_K + unit * UNIT;
      T* to = smem + (s % STAGES) * ROWS * LD + first * LD + unit * UNIT;
#pragma unroll
      for (int i = 0; i < COPIES; ++i) {
        const T* at = src[first + i * STEP];
        const bool has = at != nullptr && k < K;
        if (VEC) {
          cp_async16(to + i * STEP * LD, has ? at + k : x, has);
        } else if constexpr (std::is_same_v<T, float>) {
#pragma unroll
          for (int e = 0; e < UNIT; ++e) {
            const bool in = has && k + e < K;
            cp_async4(to + i * STEP * LD + e, in ? at + k + e : x, in);
          }
        } else {      // (2 bytes are no unit of cp.async)
          T v[UNIT];
#pragma unroll
          for (int e = 0; e < UNIT; ++e) v[e] = has && k + e < K ? __ldg(at + k + e) : from_f32<T>(0.f);
#pragma unroll
          for (int e = 0; e < UNIT; ++e) to[i * STEP * LD + e] = v[e];
        }
      }
    }
    cp_async_commit();
  };
#pragma unroll
  for (int s = 0; s < STAGES - 1; ++s) fetch(s);

  const int row0 = lane >> 3, col0 = lane & 7;
  unsigned long long pairs[MI][8];
#pragma unroll
  for (int i = 0; i < MI; ++i)
#pragma unroll
    for (int j = 0; j < 8; ++j) pairs[i][j] = 0ull;      // two zeros

  for (int s = 0; s < stages; ++s) {
    cp_async_wait<STAGES - 2>();
    __syncthreads();      // stage s is here for all; the stage before it has been read by all
    fetch(s + STAGES - 1);
    const T* xs = smem + (s % STAGES) * ROWS * LD + row0 * LD + part * PART_K;
    const T* ws = smem + (s % STAGES) * ROWS * LD + (TM + col0) * LD + part * PART_K;
    // the next row's four k's, and the columns' next, are on their way during a row's products; products of one
    // sum lie eight instructions apart
    Quad b[2][8], a[2];
#pragma unroll
    for (int j = 0; j < 8; ++j) b[0][j] = load_quad(ws + 8 * j * LD);
    a[0] = load_quad(xs);
#pragma unroll
    for (int k = 0; k < PART_K; k += 4) {
      const Quad(&now)[8] = b[(k / 4) & 1];
      Quad(&next)[8] = b[(k / 4 + 1) & 1];
#pragma unroll
      for (int i = 0; i < MI; ++i) {
        const Quad ai = a[i & 1];
        if (i + 1 < MI) a[(i + 1) & 1] = load_quad(xs + 4 * (i + 1) * LD + k);
        else if (k + 4 < PART_K) a[(i + 1) & 1] = load_quad(xs + k + 4);
        if (k + 4 < PART_K) {
#pragma unroll
          for (int j = i * 8 / MI; j < (i + 1) * 8 / MI; ++j) next[j] = load_quad(ws + 8 * j * LD + k + 4);
        }
#pragma unroll
        for (int j = 0; j < 8; ++j) fma_pair(pairs[i][j], ai.lo, now[j].lo);
#pragma unroll
        for (int j = 0; j < 8; ++j) fma_pair(pairs[i][j], ai.hi, now[j].hi);
      }
    }
  }
  float acc[MI][8];
#pragma unroll
  for (int i = 0; i < MI; ++i)
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[i][j] = sum_of_pair(pairs[i][j]);
  // (Not earlier: the next kernel's blocks would settle unevenly beside this one's, some multiprocessors taking two:
  // 300 instead of 246 us, by an earlier form of this kernel, for one after another at 517 x 896 x 4864.)
  pdl_trigger();
  // the parts' sums, a lane's in the place of its like in the other warps: (0 + 1) + (2 + 3)
  cp_async_wait<0>();
  float4* sums = reinterpret_cast<float4*>(gp_smem) + lane;
#pragma unroll
  for (int round = 0; round < 2; ++round) {
    __syncthreads();
    const bool gives = round == 0 ? (part & 1) != 0 : part == 2, takes = round == 0 ? (part & 1) == 0 : part == 0;
    float4* at = sums + (round == 0 ? part / 2 : 0) * MI * 2 * 32;
    if (gives) {
#pragma unroll
      for (int i = 0; i < MI; ++i)
#pragma unroll
        for (int q = 0; q < 2; ++q)
          at[(2 * i + q) * 32] = make_float4(acc[i][4 * q], acc[i][4 * q + 1], acc[i][4 * q + 2], acc[i][4 * q + 3]);
    }
    __syncthreads();
    if (takes) {
#pragma unroll
      for (int i = 0; i < MI; ++i)
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          const float4 v = at[(2 * i + q) * 32];
          acc[i][4 * q] += v.x, acc[i][4 * q + 1] += v.y, acc[i][4 * q + 2] += v.z, acc[i][4 * q + 3] += v.w;
        }
    }
  }
  if (part != 0) return;
#pragma unroll
  for (int i = 0; i < MI; ++i) {
    const int m = m0 + row0 + 4 * i;
    if (m >= M) continue;
    float scale = 1.f;      // a gated row of the grouped layout may count as its scale times the row
    if (GATED && row_scale != nullptr) {
      const int from = row_src[m];
      scale = from >= 0 ? row_scale[from] : 0.f;
    }
#pragma unroll
    for (int j = 0; j < (GATED ? 4 : 8); ++j) {
      const int n = n0 + col0 + 8 * j;
      if (n >= N) continue;
      float v;
      if (GATED) {
        v = gate_pair(acc[i][j] * scale, acc[i][(j + 4) % 8] * scale, gate_act, gate_limit);
      } else {
        v = acc[i][j] + (bias ? to_f32<T>(bias[n]) : 0.f);
        if (gelu) v = lab_act(v, gelu);      // the activation after the bias, before the rounding
      }
      out[(size_t)m * ldo + n] = from_f32<OutT>(v);
    }
  }
}

// Per-head products for few tokens (a decode step): out[t, h, n] = sum_k w[h, n, k] * x[t, h, k].  A warp
// forms one output column for every token: it reads the weight row once, lanes over k, and finishes each
// token's sum with a shuffle tree; the tokens' inputs of the head wait in shared memory.  The tiles above walk K in
// stages of 64 behind a barrier each, for 16 rows or more.
constexpr int HF_TOKENS = 16;
template <typename T, typename OutT>
__global__ void __launch_bounds__(256) gemm_heads_few_kernel(OutT* __restrict__ out, const T* __restrict__ x,
                                                             const T* __restrict__ w, int M, int N, int K, int ldx,
                                                             int ldo, long long head_x, long long head_o) {
  extern __shared__ float hf_x[];      // [M][K]
  pdl_trigger();
  pdl_wait();
  const int h = blockIdx.y, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int i = threadIdx.x; i < M * K; i += 256) hf_x[i] = to_f32<T>(x[(size_t)(i / K) * ldx + h * head_x + i % K]);
  __syncthreads();
  const int n = blockIdx.x * 8 + warp;
  if (n >= N) return;
  const T* row = w + ((size_t)h * N + n) * K;
  float acc[HF_TOKENS];
#pragma unroll
  for (int t = 0; t < HF_TOKENS; ++t) acc[t] = 0.f;
  for (int k = lane; k < K; k += 32) {
    const float wv = to_f32<T>(row[k]);
#pragma unroll
    for (int t = 0; t < HF_TOKENS; ++t)
      if (t < M) acc[t] = fmaf(wv, hf_x[t * K + k], acc[t]);
  }
#pragma unroll
  for (int t = 0; t < HF_TOKENS; ++t) {
    if (t >= M) break;
    const float v = warp_sum(acc[t]);
    if (lane == 0) out[(size_t)t * ldo + h * head_o + n] = from_f32<OutT>(v);
  }
}

template <typename T, typename OutT>
int launch_heads_few(void* out, const void* x, const void* w, int M, int N, int K, int ldx, int ldo, int heads,
                     long long head_x, long long head_o, cudaStream_t stream) {
  return (int)lab_launch(gemm_heads_few_kernel<T, OutT>, dim3((N + 7) / 8, heads), dim3(256),
                         sizeof(float) * (size_t)M * K, stream, (OutT*)out, (const T*)x, (const T*)w, M, N, K, ldx, ldo,
                         head_x, head_o);
}

// Grouped rows for few rows (a decode step's pairs of token and expert): the tiles above would walk K in stages
// of 64 behind a barrier each for a handful of live rows.  Here a CTA takes one tile of the layout and 16 (gated)
// or 32 output columns; a warp reads its four weight rows once, 16 bytes a lane where the rows allow it, for up
// to GF_ROWS live rows of the tile, whose inputs wait in shared memory in 32-bit; each row's sums close with a
// shuffle tree.  More live rows take further passes.  Rows whose source is -1 stay unwritten.
constexpr int GF_ROWS = 8;      // live rows a pass takes
constexpr int GF_KC = 1024;     // inputs of a row that wait in shared memory at a time
constexpr int GF_TILE_MAX = 128;

template <typename T> struct Vec16;
template <> struct Vec16<float> {
  static constexpr int N = 4;
  static __device__ __forceinline__ void load(const float* p, float* v) {
    const float4 q = *reinterpret_cast<const float4*>(p);
    v[0] = q.x; v[1] = q.y; v[2] = q.z; v[3] = q.w;
  }
};
template <> struct Vec16<__nv_bfloat16> {
  static constexpr int N = 8;
  static __device__ __forceinline__ void load(const __nv_bfloat16* p, float* v) {
    const uint4 q = *reinterpret_cast<const uint4*>(p);
    const uint32_t u[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      v[2 * i] = __uint_as_float(u[i] << 16);
      v[2 * i + 1] = __uint_as_float(u[i] & 0xffff0000u);
    }
  }
};

template <typename T, typename OutT, bool GATED>
__global__ void __launch_bounds__(256) gemm_grouped_few_kernel(OutT* __restrict__ out, const T* __restrict__ x,
                                                               const T* __restrict__ w, int M, int N, int K, int ldx,
                                                               int ldo, long long group_w,
                                                               const int* __restrict__ row_src, int row_div,
                                                               int gather, const int* __restrict__ tile_group,
                                                               int tile, int vec, int gate_act, float gate_limit,
                                                               const float* __restrict__ row_scale) {
  __shared__ float xs[GF_ROWS][GF_KC];
  __shared__ int live_row[GF_TILE_MAX], live_x[GF_TILE_MAX];
  __shared__ float live_scale[GF_TILE_MAX];      // gated: the row counts as its scale times the row
  __shared__ int n_live_s;
  pdl_trigger();
  pdl_wait();
  const int group = tile_group[blockIdx.y];
  if (group < 0) return;
  w += (long long)group * group_w;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, m0 = blockIdx.y * tile;
  // the tile's live rows in their order: a thread a row, places from the warps' ballots
  __shared__ int warp_live[GF_TILE_MAX / 32];
  const int my_src = (tid < tile && m0 + tid < M) ? row_src[m0 + tid] : -1;
  const unsigned ballot = __ballot_sync(0xffffffffu, my_src >= 0);
  if (tid < GF_TILE_MAX && lane == 0) warp_live[warp] = __popc(ballot);
  __syncthreads();
  if (tid < GF_TILE_MAX) {
    int at = __popc(ballot & ((1u << lane) - 1u)), all = 0;
#pragma unroll
    for (int i = 0; i < GF_TILE_MAX / 32; ++i) {
      if (i < warp) at += warp_live[i];
      all += warp_live[i];
    }
    if (my_src >= 0) {
      live_row[at] = m0 + tid;
      live_x[at] = gather ? my_src / row_div : m0 + tid;
      live_scale[at] = row_scale != nullptr ? row_scale[my_src] : 1.f;
    }
    if (tid == 0) n_live_s = all;
  }
  __syncthreads();
  const int n_live = n_live_s;
  // the warp's four weight rows: gate and up of two neighbouring columns, or four neighbouring columns
  constexpr int NR = 4;
  const int n0 = (blockIdx.x * 8 + warp) * (GATED ? 2 : NR);
  int col[NR];
  const T* wrow[NR];
#pragma unroll
  for (int r = 0; r < NR; ++r) {
    col[r] = GATED ? n0 + (r >> 1) : n0 + r;
    const int c = col[r] < N ? col[r] : 0;        // a row beyond the last reads row 0; its sums are dropped
    wrow[r] = w + (size_t)(GATED && (r & 1) ? N + c : c) * K;
  }
  const bool any = n0 < N;
  for (int r0 = 0; r0 < n_live; r0 += GF_ROWS) {
    const int rows = min(GF_ROWS, n_live - r0);
    float acc[NR][GF_ROWS];
#pragma unroll
    for (int r = 0; r < NR; ++r)
#pragma unroll
      for (int t = 0; t < GF_ROWS; ++t) acc[r][t] = 0.f;
    for (int k0 = 0; k0 < K; k0 += GF_KC) {
      const int kc = min(GF_KC, K - k0);
      __syncthreads();      // whoever still read the inputs before is done
      for (int t = 0; t < rows; ++t) {
        const T* src = x + (size_t)live_x[r0 + t] * ldx + k0;
        for (int k = tid; k < kc; k += 256) xs[t][k] = to_f32<T>(src[k]);
      }
      __syncthreads();
      if (!any) continue;
      if (vec) {
        constexpr int V = Vec16<T>::N;
        for (int k = lane * V; k < kc; k += 32 * V) {
          float wv[NR][V];
#pragma unroll
          for (int r = 0; r < NR; ++r) Vec16<T>::load(wrow[r] + k0 + k, wv[r]);
#pragma unroll
          for (int t = 0; t < GF_ROWS; ++t) {
            if (t < rows) {
#pragma unroll
              for (int e = 0; e < V; ++e) {
                const float xv = xs[t][k + e];
#pragma unroll
                for (int r = 0; r < NR; ++r) acc[r][t] = fmaf(wv[r][e], xv, acc[r][t]);
              }
            }
          }
        }
      } else {
        for (int k = lane; k < kc; k += 32) {
          float wv[NR];
#pragma unroll
          for (int r = 0; r < NR; ++r) wv[r] = to_f32<T>(wrow[r][k0 + k]);
#pragma unroll
          for (int t = 0; t < GF_ROWS; ++t)
            if (t < rows) {
              const float xv = xs[t][k];
#pragma unroll
              for (int r = 0; r < NR; ++r) acc[r][t] = fmaf(wv[r], xv, acc[r][t]);
            }
        }
      }
    }
    if (!any) continue;
#pragma unroll
    for (int t = 0; t < GF_ROWS; ++t) {
      if (t >= rows) break;
      float v[NR];
#pragma unroll
      for (int r = 0; r < NR; ++r) v[r] = warp_sum(acc[r][t]);
      if (lane != 0) continue;
      OutT* dst = out + (size_t)live_row[r0 + t] * ldo;
      if (GATED) {
        const float scale = live_scale[r0 + t];
#pragma unroll
        for (int c = 0; c < NR / 2; ++c)
          if (col[2 * c] < N)
            dst[col[2 * c]] = from_f32<OutT>(gate_pair(v[2 * c] * scale, v[2 * c + 1] * scale, gate_act, gate_limit));
      } else {
#pragma unroll
        for (int r = 0; r < NR; ++r)
          if (col[r] < N) dst[col[r]] = from_f32<OutT>(v[r]);
      }
    }
  }
}

template <typename T, typename OutT>
int launch_grouped_few(void* out, const void* x, const void* w, int M, int N, int K, int ldx, int ldo, int gated,
                       long long group_w, const int* row_src, int row_div, int gather, const int* tile_group, int tile,
                       cudaStream_t stream, float gate_limit, const float* row_scale) {
  constexpr int V = 16 / (int)sizeof(T);
  const int vec = K % V == 0 && ((uintptr_t)w & 15) == 0;
  const int cols = gated ? 16 : 32;      // 8 warps, four weight rows each
  dim3 grid((N + cols - 1) / cols, (M + tile - 1) / tile);
  if (gated)
    return (int)lab_launch(gemm_grouped_few_kernel<T, OutT, true>, grid, dim3(256), 0, stream, (OutT*)out, (const T*)x,
                           (const T*)w, M, N, K, ldx, ldo, group_w, row_src, row_div, gather, tile_group, tile, vec,
                           (int)(gated == 4), gate_limit, row_scale);
  return (int)lab_launch(gemm_grouped_few_kernel<T, OutT, false>, grid, dim3(256), 0, stream, (OutT*)out, (const T*)x,
                         (const T*)w, M, N, K, ldx, ldo, group_w, row_src, row_div, gather, tile_group, tile, vec, 0,
                         0.f, nullptr);
}

// Few rows of 32-bit floats (a decode step).  A warp's lanes are 8 output columns by the four parts of the sum over k; a
// lane keeps MR rows.  WR of a CTA's four warps share the rows among them, the others take further columns: few rows of
// a wide output are bound by the weights' way from memory, narrow outputs by the parts' chains of multiply-adds and the
// loads from shared memory, so a CTA takes no more columns than it must.  Rows and stages as in the tiles above.
// Measured as above: 8 x 4864 x 896 gated 14 us (113), 8 x 896 x 4864 18 us (418), 1 x 151936 x 896 84 us (606; the
// weights' way from memory takes 83); 24 x 896 x 4864 36 us, 61 in tiles of 16 rows.
constexpr int FR_ROWS = 32, FR_STAGES = 4;

template <bool GATED, int MR, int WR>
__global__ void __launch_bounds__(128) gemm_few_rows_kernel(float* __restrict__ out, const float* __restrict__ x,
                                                            const float* __restrict__ w, const float* __restrict__ bias,
                                                            int M, int N, int K, int ldx, int ldo, int act,
                                                            float gate_limit) {
  extern __shared__ __align__(16) float fr_smem[];
  constexpr int G = GATED ? 2 : 1, LD = STAGE_K + 4, COLS = 8 * (4 / WR), ROWS = G * COLS + WR * MR;
  constexpr int COPIES = (ROWS + 7) / 8;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, n0 = blockIdx.x * COLS;
  const int col = (warp / WR) * 8 + (lane & 7), part = lane >> 3, row0 = (warp % WR) * MR;
  pdl_wait();
  const int stages = (K + STAGE_K - 1) / STAGE_K;
  // a thread copies unit tid % 16 of every eighth row (weight rows, then x's)
  const int unit = tid % 16, first = tid / 16;
  const float* src[COPIES];
#pragma unroll
  for (int i = 0; i < COPIES; ++i) {
    const int row = first + 8 * i, n = n0 + row % COLS, m = row - G * COLS;
    src[i] = row < G * COLS ? (n < N ? w + (size_t)(row >= COLS ? N + n : n) * K : nullptr)
                            : (row < ROWS && m < M ? x + (size_t)m * ldx : nullptr);
  }
  auto fetch = [&](int s) {
    if (s < stages) {
      float* to = fr_smem + (s % FR_STAGES) * ROWS * LD + first * LD + unit * 4;
      const int k = s * STAGE_K + unit * 4;
#pragma unroll
      for (int i = 0; i < COPIES; ++i) {
        if (ROWS % 8 != 0 && first + 8 * i >= ROWS) break;
        const bool has = src[i] != nullptr && k < K;
        cp_async16(to + 8 * i * LD, has ? src[i] + k : x, has);
      }
    }
    cp_async_commit();
  };
#pragma unroll
  for (int s = 0; s < FR_STAGES - 1; ++s) fetch(s);
  unsigned long long pairs[G][MR];
#pragma unroll
  for (int g = 0; g < G; ++g)
#pragma unroll
    for (int i = 0; i < MR; ++i) pairs[g][i] = 0ull;      // two zeros
  for (int s = 0; s < stages; ++s) {
    cp_async_wait<FR_STAGES - 2>();
    __syncthreads();      // stage s is here for all; the stage before has been read by all
    fetch(s + FR_STAGES - 1);
    const float* base = fr_smem + (s % FR_STAGES) * ROWS * LD + part * PART_K;
    const float* wr = base + col * LD;
    const float* xr = base + (G * COLS + row0) * LD;
#pragma unroll
    for (int k = 0; k < PART_K; k += 4) {      // (entries beyond K are zeros)
      Quad wv[G], xv[MR];
#pragma unroll
      for (int g = 0; g < G; ++g) wv[g] = load_quad(wr + g * COLS * LD + k);
#pragma unroll
      for (int i = 0; i < MR; ++i) xv[i] = load_quad(xr + i * LD + k);
#pragma unroll
      for (int g = 0; g < G; ++g)
#pragma unroll
        for (int i = 0; i < MR; ++i) fma_pair(pairs[g][i], xv[i].lo, wv[g].lo);
#pragma unroll
      for (int g = 0; g < G; ++g)
#pragma unroll
        for (int i = 0; i < MR; ++i) fma_pair(pairs[g][i], xv[i].hi, wv[g].hi);
    }
  }
  pdl_trigger();
  cp_async_wait<0>();
  const int n = n0 + col;
#pragma unroll
  for (int i = 0; i < MR; ++i) {
    float t[G];
#pragma unroll
    for (int g = 0; g < G; ++g) {      // (0 + 1) + (2 + 3): both partners form the same sum
      t[g] = sum_of_pair(pairs[g][i]);
      t[g] += __shfl_xor_sync(0xffffffffu, t[g], 8);
      t[g] += __shfl_xor_sync(0xffffffffu, t[g], 16);
    }
    const int m = row0 + i;
    if (m >= M || n >= N || part != 0) continue;
    float v;
    if (GATED) {
      v = gate_pair(t[0], t[G - 1], act, gate_limit);
    } else {
      v = t[0] + (bias ? bias[n] : 0.f);
      if (act) v = lab_act(v, act);
    }
    out[(size_t)m * ldo + n] = v;
  }
}

template <bool GATED, int MR, int WR>
int launch_few_rows_as(void* out, const void* x, const void* w, const void* bias, int M, int N, int K, int ldx, int ldo,
                       int act, float gate_limit, cudaStream_t stream) {
  constexpr int cols = 8 * (4 / WR);
  const size_t smem = sizeof(float) * FR_STAGES * ((GATED ? 2 : 1) * cols + WR * MR) * (STAGE_K + 4);
  static LabShared granted;
  const cudaError_t e = lab_allow_shared(granted, (const void*)gemm_few_rows_kernel<GATED, MR, WR>, smem);
  if (e != cudaSuccess) return (int)e;
  return (int)lab_launch(gemm_few_rows_kernel<GATED, MR, WR>, dim3((N + cols - 1) / cols), dim3(128), smem, stream,
                         (float*)out, (const float*)x, (const float*)w, (const float*)bias, M, N, K, ldx, ldo, act,
                         gate_limit);
}

inline int launch_few_rows(void* out, const void* x, const void* w, const void* bias, int M, int N, int K, int ldx,
                           int ldo, bool gate, int act, float gate_limit, cudaStream_t stream) {
#define LAB_FEW(MR_, WR_)                                                                                            \
  return (gate ? launch_few_rows_as<true, MR_, WR_> : launch_few_rows_as<false, MR_, WR_>)(                          \
      out, x, w, gate ? nullptr : bias, M, N, K, ldx, ldo, act, gate_limit, stream)
  if (M <= 2) LAB_FEW(2, 1);
  if (M <= 4) LAB_FEW(2, 2);
  if (M <= 8) LAB_FEW(2, 4);
  if (M <= 16) LAB_FEW(4, 4);
  LAB_FEW(8, 4);
#undef LAB_FEW
}

template <typename T, typename OutT, bool GATED, int MI, bool VEC>
int launch_tile(void* out, const void* x, const void* w, const void* bias, int M, int N, int K, int ldx, int ldo, int act,
                cudaStream_t stream, int batch, long long batch_x, long long batch_w, long long batch_o,
                const int* row_src, int row_div, const int* tile_group, float gate_limit, const float* row_scale) {
  using Shape = TileShape<T, MI>;
  constexpr int cols = GATED ? Shape::COLS / 2 : Shape::COLS;
  const auto kernel = gemm_plain_kernel<T, OutT, GATED, MI, VEC>;
  static LabShared granted;
  const cudaError_t e = lab_allow_shared(granted, (const void*)kernel, Shape::BYTES);
  if (e != cudaSuccess) return (int)e;
  constexpr int most = 65534 * Shape::ROWS;      // rows of a launch: the grid's limit, whole tiles of groups
  for (int m0 = 0; m0 < M; m0 += most) {
    const int rows = M - m0 < most ? M - m0 : most;
    const dim3 grid((N + cols - 1) / cols, (rows + Shape::ROWS - 1) / Shape::ROWS, batch);
    const cudaError_t f = lab_launch(
        kernel, grid, dim3(Shape::THREADS), Shape::BYTES, stream, (OutT*)out + (size_t)m0 * ldo,
        (const T*)x + (row_src == nullptr ? (size_t)m0 * ldx : 0), (const T*)w, (const T*)bias, rows, N, K, ldx, ldo, batch_x,
        batch_w, batch_o, GATED ? 0 : act, row_src == nullptr ? nullptr : row_src + m0, row_div,
        tile_group == nullptr ? nullptr : tile_group + m0 / BM, GATED ? act : 0, gate_limit, row_scale);
    if (f != cudaSuccess) return (int)f;
    if (M - m0 <= most) break;
  }
  return 0;
}

// Whether tiles of 16 rows serve M rows of N accumulator columns, rather than tiles of 32.  A launch takes as long as the
// multiprocessor with the most tiles, and a tile of 16 rows costs 0.54 of one of 32 (measured: 0.49 where a
// multiprocessor has one, 0.57 where it has four).  517 x 896 x 4864: 155 us in tiles of 32, 176 of 16; 517 x 1152 x 896:
// 47 and 43; 100 x 896 x 4864: 93 and 74.
static inline bool flat_tiles(long long M, long long N, int batch) {
  const long long columns = (N + 63) / 64 * batch, sms = lab_sm_count();
  return ((M + 15) / 16 * columns + sms - 1) / sms * 54 < ((M + 31) / 32 * columns + sms - 1) / sms * 100;
}

template <typename T, typename OutT>
int launch(void* out, const void* x, const void* w, const void* bias, int M, int N, int K, int ldx, int ldo, int gated,
           cudaStream_t stream, int batch = 1, long long batch_x = 0, long long batch_w = 0, long long batch_o = 0,
           const int* row_src = nullptr, int row_div = 1, const int* tile_group = nullptr, float gate_limit = 0.f,
           const float* row_scale = nullptr) {
  const bool gate = gated == 1 || gated == 4;
  const int act = gate ? (int)(gated == 4) : (gated >= 2 ? gated - 1 : 0);
  constexpr int unit = 16 / (int)sizeof(T);
  const bool units = K % unit == 0 && ldx % unit == 0 && batch_x % unit == 0 && batch_w % unit == 0 &&
                     (((uintptr_t)x | (uintptr_t)w) & 15) == 0;
  if constexpr (std::is_same_v<T, float>) {
    if (batch == 1 && row_src == nullptr && tile_group == nullptr && f32_on_tensor_cores(N, K, gate))
      return launch_f32(out, x, w, bias, M, N, K, ldx, ldo, gate, act, gate_limit, stream);
    if (M <= FR_ROWS && batch == 1 && row_src == nullptr && tile_group == nullptr && units)
      return launch_few_rows(out, x, w, bias, M, N, K, ldx, ldo, gate, act, gate_limit, stream);
  }
  const bool flat = tile_group == nullptr && flat_tiles(M, gate ? 2ll * N : N, batch);
#define LAB_TILE(GATED_, MI_)                                                                                       \
  return (units ? launch_tile<T, OutT, GATED_, MI_, true> : launch_tile<T, OutT, GATED_, MI_, false>)(              \
      out, x, w, gate ? nullptr : bias, M, N, K, ldx, ldo, act, stream, batch, batch_x, batch_w, batch_o, row_src,  \
      row_div, tile_group, gate_limit, gate ? row_scale : nullptr)
  if (gate && flat) LAB_TILE(true, 4);
  if (gate) LAB_TILE(true, 8);
  if (flat) LAB_TILE(false, 4);
  LAB_TILE(false, 8);
#undef LAB_TILE
}
}  // namespace

// N is the number of output columns; with gated == 1, w holds 2 N rows (gate rows, then up rows); gated == 2 is
// the plain product with GELU (tanh form) after the bias, 3 with the square of relu; 4 is the pair gated by the tanh
// form of GELU (2 N rows as well).
LAB_EXPORT int lab_gemm_plain(void* out, const void* x, const void* w, const void* bias, int M, int N, int K, int ldx,
                              int ldo, int gated, int dtype, int out_f32, float gate_limit, cudaStream_t stream) {
  if (M <= 0 || N <= 0) return 0;
  if (dtype == LAB_F32)
    return launch<float, float>(out, x, w, bias, M, N, K, ldx, ldo, gated, stream, 1, 0, 0, 0, nullptr, 1, nullptr, gate_limit);
  if (out_f32)
    return launch<__nv_bfloat16, float>(out, x, w, bias, M, N, K, ldx, ldo, gated, stream, 1, 0, 0, 0, nullptr, 1, nullptr,
                                        gate_limit);
  return launch<__nv_bfloat16, __nv_bfloat16>(out, x, w, bias, M, N, K, ldx, ldo, gated, stream, 1, 0, 0, 0, nullptr, 1,
                                              nullptr, gate_limit);
}

// `batch` products of one shape in one launch: out_b[m, n] = sum_k x_b[m, k] * w_b[n, k], operand b lying
// b * batch_* elements after operand 0 (heads side by side in a row: batch_x = the head's width).
LAB_EXPORT int lab_gemm_plain_batched(void* out, const void* x, const void* w, int M, int N, int K, int ldx, int ldo,
                                      int batch, long long batch_x, long long batch_w, long long batch_o, int dtype,
                                      int out_f32, cudaStream_t stream) {
  if (M <= 0 || N <= 0 || batch <= 0) return 0;
  if (batch > 65535) return (int)cudaErrorInvalidValue;
  if (M <= HF_TOKENS && (size_t)M * K * sizeof(float) <= 48 * 1024 && batch_w == (long long)N * K) {
    if (dtype == LAB_F32)
      return launch_heads_few<float, float>(out, x, w, M, N, K, ldx, ldo, batch, batch_x, batch_o, stream);
    if (out_f32)
      return launch_heads_few<__nv_bfloat16, float>(out, x, w, M, N, K, ldx, ldo, batch, batch_x, batch_o, stream);
    return launch_heads_few<__nv_bfloat16, __nv_bfloat16>(out, x, w, M, N, K, ldx, ldo, batch, batch_x, batch_o, stream);
  }
  if (dtype == LAB_F32)
    return launch<float, float>(out, x, w, nullptr, M, N, K, ldx, ldo, 0, stream, batch, batch_x, batch_w, batch_o);
  if (out_f32)
    return launch<__nv_bfloat16, float>(out, x, w, nullptr, M, N, K, ldx, ldo, 0, stream, batch, batch_x, batch_w,
                                        batch_o);
  return launch<__nv_bfloat16, __nv_bfloat16>(out, x, w, nullptr, M, N, K, ldx, ldo, 0, stream, batch, batch_x, batch_w,
                                              batch_o);
}

// Rows grouped by the matrix they meet (routed experts): tile t of lab_gemm_plain_group_rows() rows meets the
// matrix tile_group[t] of `w` (matrices group_w elements apart; -1: the tile holds no rows and is skipped); row m of
// the product reads x's row row_src[m] / row_div (row_src null: row m itself; -1: padding, read as zeros).
// M counts the rows of the grouped layout (out has that many); x must hold every row that row_src names.
// row_scale (gated; null: none): the product of row m is that of row_scale[row_src[m]] times the row.
LAB_EXPORT int lab_gemm_plain_group_rows() { return BM; }
LAB_EXPORT int lab_gemm_plain_grouped(void* out, const void* x, const void* w, int M, int N, int K, int ldx, int ldo,
                                      int gated, long long group_w, const int* row_src, int row_div,
                                      const int* tile_group, int dtype, int out_f32, float gate_limit,
                                      const float* row_scale, cudaStream_t stream) {
  if (M <= 0 || N <= 0) return 0;
  if (row_scale != nullptr && (!gated || row_src == nullptr)) return (int)cudaErrorInvalidValue;
  if (tile_group == nullptr || row_div < 1) return (int)cudaErrorInvalidValue;
  if (dtype == LAB_F32)
    return launch<float, float>(out, x, w, nullptr, M, N, K, ldx, ldo, gated, stream, 1, 0, group_w, 0, row_src, row_div,
                                tile_group, gate_limit, row_scale);
  if (out_f32)
    return launch<__nv_bfloat16, float>(out, x, w, nullptr, M, N, K, ldx, ldo, gated, stream, 1, 0, group_w, 0, row_src,
                                        row_div, tile_group, gate_limit, row_scale);
  return launch<__nv_bfloat16, __nv_bfloat16>(out, x, w, nullptr, M, N, K, ldx, ldo, gated, stream, 1, 0, group_w, 0,
                                              row_src, row_div, tile_group, gate_limit, row_scale);
}

// The same product for few rows (a decode step): tile t of `tile` rows (at most 128) meets matrix tile_group[t];
// only rows whose row_src is not -1 are formed and written.  gather: row m reads x's row row_src[m] / row_div,
// else x's row m.
LAB_EXPORT int lab_gemm_plain_grouped_few(void* out, const void* x, const void* w, int M, int N, int K, int ldx,
                                          int ldo, int gated, long long group_w, const int* row_src, int row_div,
                                          int gather, const int* tile_group, int tile, int dtype, int out_f32,
                                          float gate_limit, const float* row_scale, cudaStream_t stream) {
  if (M <= 0 || N <= 0) return 0;
  if (tile_group == nullptr || row_src == nullptr || row_div < 1 || tile < 1 || tile > GF_TILE_MAX || K <= 0)
    return (int)cudaErrorInvalidValue;
  if ((M + tile - 1) / tile > 65535) return (int)cudaErrorInvalidValue;
  if (dtype == LAB_F32)
    return launch_grouped_few<float, float>(out, x, w, M, N, K, ldx, ldo, gated, group_w, row_src, row_div, gather,
                                            tile_group, tile, stream, gate_limit, row_scale);
  if (out_f32)
    return launch_grouped_few<__nv_bfloat16, float>(out, x, w, M, N, K, ldx, ldo, gated, group_w, row_src, row_div,
                                                    gather, tile_group, tile, stream, gate_limit, row_scale);
  return launch_grouped_few<__nv_bfloat16, __nv_bfloat16>(out, x, w, M, N, K, ldx, ldo, gated, group_w, row_src,
                                                          row_div, gather, tile_group, tile, stream, gate_limit,
                                                          row_scale);
}
