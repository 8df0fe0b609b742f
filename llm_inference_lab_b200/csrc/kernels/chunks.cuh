// A recurrence over a matrix state in chunks of rows side by side.  A request's chunks of 64 rows start at its first row;
// once the state before each chunk is known, its outputs are
//
//     o_i = G_i S^T q_i + sum_{j<=i} g_ij s_j (q_i . k_j) v_j
//
// with G_i the product of the chunk's decays up to row i and g_ij that of the decays after row j up to row i: products of
// small matrices in 32-bit.  Products of decays are formed as products, never as quotients, so strong decays lose nothing,
// and no output touches a later row.
#pragma once
#include "common.cuh"

namespace {

// SiLU by the hardware's 2^x and reciprocal approximations (relative error about 2^-21, as the attention
// kernels' softmax has it): a few instructions instead of the seventy of the exact exponential and division,
// which the recurrence's helpers would otherwise spend longer on than its walkers on their chunk.
__device__ __forceinline__ float silu_quick(float z) { return __fdividef(z, 1.0f + fast_exp2(-1.4426950408889634f * z)); }

constexpr int CHUNK = 64, WIDE = 72;      // rows of a chunk; columns of a slice of V at most
constexpr int CHUNK_THREADS = 160;        // 8 x up to 18 tiles of 8 x 4, and the rest of the last warp

// The place of a request's first chunk: there are no more than tokens / 64 + requests.
__host__ __device__ __forceinline__ int first_chunk(int row0, int request) { return row0 / CHUNK + request; }

// The request whose chunk lies at `at`, the chunk's first row and its rows (0: nobody's place).
__device__ __forceinline__ int chunk_rows(const int* q_start, const int* state_slot, int requests, int n_slots, int at, int& row0,
                                          int& rows) {
  const int lane = threadIdx.x & 31;
  int r = 0;
  for (int r0 = 0; r0 < requests; r0 += 32) {
    const bool before = r0 + lane < requests && first_chunk(q_start[min(r0 + lane, requests - 1)], r0 + lane) <= at;
    const unsigned all = __ballot_sync(0xffffffffu, before);
    if (all == 0u) break;
    r = r0 + 31 - __clz((int)all);
  }
  const int first = q_start[r];
  row0 = first + CHUNK * (at - first_chunk(first, r));
  rows = max(0, min(CHUNK, q_start[r + 1] - row0));
  if (state_slot[r] < 0 || state_slot[r] >= n_slots) rows = 0;      // padding; the kernel between reports the others
  return r;
}

// A thread's tile of 8 rows and 4 columns: pairs of rows, two multiply-adds an instruction.
struct Tile {
  f32x2 at[4][4];      // [pair of rows][column]
  __device__ __forceinline__ void clear() {
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) at[i][j] = 0ull;
  }
  // one step of k: rows 0..3 of A at a0, 4..7 at a1, B's four columns at b
  __device__ __forceinline__ void step(const float* a0, const float* a1, const float* b) {
    const ulonglong2 x = *reinterpret_cast<const ulonglong2*>(a0), y = *reinterpret_cast<const ulonglong2*>(a1);
    const float4 z = load4(b);
    const f32x2 a[4] = {x.x, x.y, y.x, y.y}, c[4] = {pair_of(z.x, z.x), pair_of(z.y, z.y), pair_of(z.z, z.z), pair_of(z.w, z.w)};
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) at[i][j] = fma2(a[i], c[j], at[i][j]);
  }
  __device__ __forceinline__ void add(const Tile& t) {
    const f32x2 one = pair_of(1.f, 1.f);
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) at[i][j] = fma2(t.at[i][j], one, at[i][j]);
  }
  __device__ __forceinline__ float get(int row, int col) const { return row % 2 ? high_of(at[row / 2][col]) : low_of(at[row / 2][col]); }
  __device__ __forceinline__ void scale(int pair, f32x2 f) {
#pragma unroll
    for (int j = 0; j < 4; ++j) at[pair][j] = mul2(at[pair][j], f);
  }
};
// Sums go in runs of 8 terms, which are then added up: a sum's roundings grow with its terms.
constexpr int RUN = 8;

// e / q and the rest for e < 65536 / q, by a multiplication
struct Divider {
  int q;
  unsigned m;
  __device__ __forceinline__ explicit Divider(int q_) : q(q_), m(65536u / q_ + 1) {}
  __device__ __forceinline__ int over(int e) const { return (int)(((unsigned)e * m) >> 16); }
  __device__ __forceinline__ int rest(int e) const { return e - over(e) * q; }
};

__device__ __forceinline__ float4 act4(float4 z, int act) {
  if (act) z.x = silu_quick(z.x), z.y = silu_quick(z.y), z.z = silu_quick(z.z), z.w = silu_quick(z.w);
  return z;
}
// four neighbouring entries, zeros beyond `count`; VEC: on 16 bytes, `count` a multiple of four
template <bool VEC>
__device__ __forceinline__ float4 row4(const float* src, int at, int count) {
  if (VEC) return at < count ? load4(src + at) : make_float4(0.f, 0.f, 0.f, 0.f);
  return make_float4(at < count ? src[at] : 0.f, at + 1 < count ? src[at + 1] : 0.f, at + 2 < count ? src[at + 2] : 0.f,
                     at + 3 < count ? src[at + 3] : 0.f);
}

// load(e) for every e below `total`, store(e, .) of what it gave: a thread's next four on their way together.
template <typename Load, typename Store>
__device__ __forceinline__ void copy_quads(int total, Load load, Store store) {
  for (int e0 = threadIdx.x; e0 < total; e0 += 4 * CHUNK_THREADS) {
    float4 z[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) z[i] = e0 + i * CHUNK_THREADS < total ? load(e0 + i * CHUNK_THREADS) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int i = 0; i < 4; ++i)
      if (e0 + i * CHUNK_THREADS < total) store(e0 + i * CHUNK_THREADS, z[i]);
  }
}

// Queries and keys lie by channel in shared memory, quads of rows at (quad of rows) ^ (quad of channels), which spreads both
// the transposing stores and the loads over the banks.
__device__ __forceinline__ int by_channel(int n, int quad) { return n * CHUNK + ((quad ^ (n / 4)) & 15) * 4; }
__device__ __forceinline__ void store_by_channel(float* base, int t, int n, float4 z) {
  float* to = base + by_channel(n, t / 4) + t % 4;
  to[0] = z.x, to[CHUNK] = z.y, to[2 * CHUNK] = z.z, to[3 * CHUNK] = z.w;
}

// tile = A^T B over `quads` quads of k: A by channel, rows 8 rg ..; B by channel, rows 4 jq ..
__device__ __forceinline__ void tile_by_channel(Tile& tile, const float* A, const float* B, int rg, int jq, int quads) {
  tile.clear();
  for (int k0 = 0; k0 < quads; k0 += RUN / 4) {
    Tile part;
    part.clear();
#pragma unroll 2
    for (int n4 = k0; n4 < min(quads, k0 + RUN / 4); ++n4) {
      const int swz = n4 & 15;
      const float *a = A + n4 * 4 * CHUNK, *b = B + n4 * 4 * CHUNK + (jq ^ swz) * 4;
#pragma unroll
      for (int m = 0; m < 4; ++m) part.step(a + m * CHUNK + ((2 * rg) ^ swz) * 4, a + m * CHUNK + ((2 * rg + 1) ^ swz) * 4, b + m * CHUNK);
    }
    tile.add(part);
  }
}

// A tile of products of rows 8 rg .. with rows j 4 jq .. (as far as j <= i), times g_ij s_j, to `to` by the row j.
__device__ __forceinline__ void store_decayed(float* to, const Tile& tile, const float* decay, const float* scale, int rg, int jq) {
  const int r0 = 8 * rg, j0 = 4 * jq;
  float between = 1.f, a[8];      // the decays after the four j's up to the rows
#pragma unroll
  for (int q = 0; q < CHUNK / 4; ++q) {
    const float4 d = load4(decay + 4 * q);
    if (q > jq && q < 2 * rg) between *= (d.x * d.y) * (d.z * d.w);
  }
#pragma unroll
  for (int i = 0; i < 8; ++i) a[i] = decay[r0 + i];
#pragma unroll
  for (int j = 3; j >= 0; --j) {
    const bool left = j0 + j < r0;
    float run = left ? between : 1.f;
    if (left) between *= decay[j0 + j];
    const float s = scale[j0 + j];
    float w[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      if (r0 + i > j0 + j) run *= a[i];
      w[i] = tile.get(i, j) * (run * s);
    }
    float* row = to + (j0 + j) * CHUNK;
    store4(row + (((2 * rg) ^ jq) & 15) * 4, make_float4(w[0], w[1], w[2], w[3]));
    store4(row + (((2 * rg + 1) ^ jq) & 15) * 4, make_float4(w[4], w[5], w[6], w[7]));
  }
}

struct ChunkParams {
  float* out;            // [tokens, ld_o]: head h at h * V
  int ld_o;
  const float* q;        // [tokens, ld_qk]: group g at g * N
  const float* k;
  int ld_qk;
  const float* v;        // [tokens, ld_v]: head h at h * V
  int ld_v;
  const float* a;        // decays: row t, head h at t * a_row + h * a_head
  size_t a_row, a_head;
  const float* s;        // scales likewise, or null (1)
  const float* states;   // [places, H, N, V]: the state before each chunk
  const int* q_start;
  const int* state_slot;
  int requests, n_slots, H, G, N, V, act;
  int vec;               // everything may be read and written 16 bytes at a time

  __device__ __forceinline__ const float* decay_of(int t, int h) const { return a + t * a_row + h * a_head; }
  // four channels of a row of q or k
  template <bool VEC>
  __device__ __forceinline__ float4 channels(const float* m, int t, int g, int n) const {
    return row4<VEC>(m + (size_t)t * ld_qk + g * N, n, N);
  }
};

// grid (places of chunks, heads, slices of V of Vs).  Bound by instructions: a row and head want 2 N V + 64 (N + V) / 2 of the
// multiply-adds, two to an instruction and a thread's 32 behind three 16-byte loads, and two others go with each; the copies
// and the transposing of q and k (a sixth of the time) wait for memory.  Queries and keys lie by channel, and the weights and
// the values take the keys' and the state's place: 53 KB for 64 channels, so that four CTAs find room on a multiprocessor and
// 2,048 rows of 14 heads all at once.
template <bool VEC>
__global__ void __launch_bounds__(CHUNK_THREADS, 4) chunk_output_kernel(ChunkParams p, int Vs) {
  extern __shared__ __align__(16) float smem[];
  pdl_wait();
  const int at = blockIdx.x, h = blockIdx.y, g = h / (p.H / p.G), tid = threadIdx.x;
  const int col0 = blockIdx.z * Vs, cols = min(Vs, p.V - col0), quads = (cols + 3) / 4, n_quads = (p.N + 3) / 4;
  int row0, rows;
  chunk_rows(p.q_start, p.state_slot, p.requests, p.n_slots, at, row0, rows);
  if (rows == 0) return;
  const int side = max(n_quads * 4, CHUNK);           // channels, later rows of the weights or the values
  float* qs = smem;                                   // [4 n_quads][64]
  float* ks = qs + n_quads * 4 * CHUNK;               // [side][64], then the rows' weights by the other row
  float* ss = ks + side * CHUNK;                      // [side][WIDE]: the state before, then the values
  float* decay = ss + side * WIDE;                    // [64], then the scales
  float* scale = decay + CHUNK;
  if (tid < CHUNK) {
    decay[tid] = tid >= rows ? 1.f : *p.decay_of(row0 + tid, h);
    scale[tid] = tid >= rows ? 0.f : p.s != nullptr ? p.s[(row0 + tid) * p.a_row + h * p.a_head] : 1.f;
  }
  const float4 zeros = make_float4(0.f, 0.f, 0.f, 0.f);
  const Divider by_n(n_quads), by_c(quads);
  auto row = [&](const float* m) {
    return [&, m](int e) { return by_n.over(e) < rows ? p.channels<VEC>(m, row0 + by_n.over(e), g, 4 * by_n.rest(e)) : zeros; };
  };
  copy_quads(CHUNK * n_quads, row(p.q), [&](int e, float4 z) { store_by_channel(qs, by_n.over(e), 4 * by_n.rest(e), act4(z, p.act)); });
  copy_quads(CHUNK * n_quads, row(p.k), [&](int e, float4 z) { store_by_channel(ks, by_n.over(e), 4 * by_n.rest(e), act4(z, p.act)); });
  const float* open = p.states + ((size_t)at * p.H + h) * p.N * p.V + col0;
  auto to_rows = [&](int e, float4 z) { store4(ss + by_c.over(e) * WIDE + 4 * by_c.rest(e), z); };
  copy_quads(n_quads * 4 * quads, [&](int e) {
    return by_c.over(e) < p.N ? row4<VEC>(open + (size_t)by_c.over(e) * p.V, 4 * by_c.rest(e), cols) : zeros;
  }, to_rows);
  __syncthreads();
  // q_i . k_j for rows 8 rg .. and j 4 quad .., as far as j <= i
  {
    const int rg = tid / 16, jq = tid % 16;
    const bool pairs = tid < 128 && 4 * jq < 8 * rg + 8;
    Tile w;
    if (pairs) tile_by_channel(w, qs, ks, rg, jq, n_quads);
    __syncthreads();      // the keys have been read
    if (pairs) store_decayed(ks, w, decay, scale, rg, jq);
  }
  // the old state's part
  const int og = by_c.over(tid), oc = by_c.rest(tid) * 4, i0 = 8 * og;
  const bool live = og < CHUNK / 8 && i0 < rows;
  Tile o;
  if (live) {
    o.clear();
    for (int k0 = 0; k0 < n_quads; k0 += RUN / 4) {
      Tile part;
      part.clear();
#pragma unroll 2
      for (int n4 = k0; n4 < min(n_quads, k0 + RUN / 4); ++n4) {
        const int swz = n4 & 15;
        const float *a = qs + n4 * 4 * CHUNK, *b = ss + n4 * 4 * WIDE + oc;
#pragma unroll
        for (int m = 0; m < 4; ++m) part.step(a + m * CHUNK + ((2 * og) ^ swz) * 4, a + m * CHUNK + ((2 * og + 1) ^ swz) * 4, b + m * WIDE);
      }
      o.add(part);
    }
    float G = 1.f;
#pragma unroll
    for (int q = 0; q < CHUNK / 4; ++q) {
      const float4 d = load4(decay + 4 * q);
      if (q < 2 * og) G *= (d.x * d.y) * (d.z * d.w);
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float g0 = G * decay[i0 + 2 * i], g1 = g0 * decay[i0 + 2 * i + 1];
      o.scale(i, pair_of(g0, g1));
      G = g1;
    }
  }
  __syncthreads();      // the state has been read
  copy_quads(CHUNK * quads, [&](int e) {
    return by_c.over(e) < rows ? row4<VEC>(p.v + (size_t)(row0 + by_c.over(e)) * p.ld_v + h * p.V + col0, 4 * by_c.rest(e), cols) : zeros;
  }, [&](int e, float4 z) { to_rows(e, act4(z, p.act)); });
  __syncthreads();
  if (!live) return;
  for (int t0 = 0; t0 < i0; t0 += RUN) {
    Tile part;
    part.clear();
#pragma unroll 4
    for (int t = t0; t < min(i0, t0 + RUN); ++t) {
      const float* a = ks + t * CHUNK;
      const int swz = t / 4;
      part.step(a + ((2 * og) ^ swz) * 4, a + ((2 * og + 1) ^ swz) * 4, ss + t * WIDE + oc);
    }
    o.add(part);
  }
  // the tile's own rows: row i takes those up to itself
  float own[8][4] = {};
#pragma unroll
  for (int t = 0; t < 8; ++t) {
    const float* a = ks + (i0 + t) * CHUNK;
    const int swz = (i0 + t) / 4;
    const float4 a0 = load4(a + ((2 * og) ^ swz) * 4), a1 = load4(a + ((2 * og + 1) ^ swz) * 4), b = load4(ss + (i0 + t) * WIDE + oc);
    const float x[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w}, c[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
    for (int i = t; i < 8; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) own[i][j] = fmaf(x[i], c[j], own[i][j]);
  }
  float* dst = p.out + (size_t)(row0 + i0) * p.ld_o + h * p.V + col0 + oc;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    if (i0 + i >= rows) break;
    float z[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) z[j] = o.get(i, j) + own[i][j];
    if (VEC) store4(dst + (size_t)i * p.ld_o, make_float4(z[0], z[1], z[2], z[3]));
    else
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (oc + j < cols) dst[(size_t)i * p.ld_o + j] = z[j];
  }
}

// Columns of a slice of V.
inline int chunk_slice(int V) {
  const int slices = (V + WIDE - 1) / WIDE;
  return ((V + slices - 1) / slices + 3) / 4 * 4;
}

inline int launch_chunk_outputs(const ChunkParams& p, int tokens, cudaStream_t stream) {
  const int channels = (p.N + 3) / 4 * 4, side = channels > CHUNK ? channels : CHUNK, Vs = chunk_slice(p.V);
  const size_t smem = (size_t)(channels * CHUNK + side * (CHUNK + WIDE) + 2 * CHUNK) * sizeof(float);
  auto launch = [&](auto kernel, LabShared& granted) {
    const cudaError_t e = lab_allow_shared(granted, (const void*)kernel, smem);
    if (e != cudaSuccess) return (int)e;
    return (int)lab_launch(kernel, dim3(first_chunk(tokens, p.requests), p.H, (p.V + Vs - 1) / Vs), dim3(CHUNK_THREADS), smem, stream,
                           p, Vs);
  };
  static LabShared wide, narrow;
  return p.vec && p.ld_o % 4 == 0 ? launch(chunk_output_kernel<true>, wide) : launch(chunk_output_kernel<false>, narrow);
}

}  // namespace
